// calculator.cu -- host orchestration of one device-resident pruning store
// and the C ABI declared in include/b3g.h.
#include "calculator.hpp"
#include "host_fold.hpp"
#include "host_math.hpp"

#include <cmath>
#include <cstring>
#include <algorithm>
#include <cstdlib>
#include <new>

namespace b3g {

void check_cuda(cudaError_t e, const char *what)
{
	if (e == cudaSuccess)
		return;
	const b3g_status s = e == cudaErrorMemoryAllocation
				     ? B3G_ERR_OUT_OF_MEMORY
				     : B3G_ERR_CUDA;
	throw Error(s, std::string(what) + ": " + cudaGetErrorString(e));
}

namespace {

size_t align_up(size_t x, size_t a) { return (x + a - 1) / a * a; }

struct DeviceGuard {
	int prev = -1;
	explicit DeviceGuard(int dev)
	{
		check_cuda(cudaGetDevice(&prev), "cudaGetDevice");
		if (prev != dev)
			check_cuda(cudaSetDevice(dev), "cudaSetDevice");
	}
	~DeviceGuard()
	{
		int cur = -1;
		if (cudaGetDevice(&cur) == cudaSuccess && cur != prev && prev >= 0)
			cudaSetDevice(prev);
	}
};

template <typename T> void dev_alloc(T *&p, size_t bytes, const char *what)
{
	void *v = nullptr;
	check_cuda(cudaMalloc(&v, bytes ? bytes : 1), what);
	p = static_cast<T *>(v);
}

// EditBuf::set_edited (sk/src/editbuf.rs:71-81)
inline void set_edited(uint8_t &m)
{
	if (!(m & 2u))
		m = static_cast<uint8_t>(((m & 1u) ^ 1u) | 2u);
}

} // namespace

Calculator::Calculator(const b3g_config &cfg, const uint8_t *samples)
{
	if (cfg.num_leaves < 2)
		throw Error(B3G_ERR_INVALID_ARGUMENT, "num_leaves must be >= 2");
	if (cfg.num_patterns < 1)
		throw Error(B3G_ERR_INVALID_ARGUMENT, "num_patterns must be >= 1");
	if (cfg.num_states != 4 && cfg.num_states != 20)
		throw Error(B3G_ERR_INVALID_ARGUMENT,
			    "num_states must be 4 (DNA) or 20 (protein)");
	if (cfg.num_states == 20 && cfg.num_categories > 8)
		throw Error(B3G_ERR_INVALID_ARGUMENT,
			    "20-state calculators take at most 8 categories");
	if (cfg.num_categories < 1 || cfg.num_categories > kMaxCategories)
		throw Error(B3G_ERR_INVALID_ARGUMENT,
			    "num_categories must be in 1..16");
	if (cfg.precision != B3G_PRECISION_F64 &&
	    cfg.precision != B3G_PRECISION_F32)
		throw Error(B3G_ERR_INVALID_ARGUMENT, "unknown precision");
	if (cfg.reserved != 0)
		throw Error(B3G_ERR_INVALID_ARGUMENT, "reserved must be 0");
	if (!samples)
		throw Error(B3G_ERR_INVALID_ARGUMENT, "samples is null");
	if (cfg.num_leaves > (1u << 24) || cfg.num_patterns > (1u << 28))
		throw Error(B3G_ERR_INVALID_ARGUMENT, "problem too large");

	L_ = cfg.num_leaves;
	I_ = L_ - 1;
	P_ = cfg.num_patterns;
	S_ = cfg.num_states;
	C_ = cfg.num_categories;
	f32_ = cfg.precision == B3G_PRECISION_F32;
	scale_ln_ = cfg.scale_ln;
	for (uint32_t d = 0; d < kScalePow; ++d)
		scale_pow_[d] = std::exp(-static_cast<double>(scale_ln_) * (d + 1));
	device_ = cfg.device;
	ldp_ = static_cast<uint32_t>(align_up(P_, kPatternAlign));
	// patterns per block: 128 threads for up to 4 categories, one warp of
	// patterns per category above that (at most 16 x 32 = 512 threads)
	tile_ = C_ <= 1 ? 128 : C_ == 2 ? 64 : 32;

	int ndev = 0;
	check_cuda(cudaGetDeviceCount(&ndev), "cudaGetDeviceCount");
	if (device_ < 0 || device_ >= ndev)
		throw Error(B3G_ERR_INVALID_ARGUMENT, "no such CUDA device");
	DeviceGuard g(device_);
	int sms = 0;
	check_cuda(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount,
					  device_),
		   "SM count");
	num_sms_ = static_cast<uint32_t>(sms);
	// run-synchronous FP32 walk: 64 patterns x C categories per tile while
	// a tile's columns fit one 512-thread block
	runs_tile_ = 64;
	while (runs_tile_ > 32 && runs_tile_ * C_ > 512)
		runs_tile_ >>= 1;
	if (const char *env = std::getenv("B3G_RUNS_TILE")) {
		const uint32_t t = static_cast<uint32_t>(std::atoi(env));
		if (t == 16 || t == 32 || t == 64 || t == 128)
			runs_tile_ = t;
	}
	if (const char *env = std::getenv("B3G_RUNS_BLOCK")) {
		const uint32_t b = static_cast<uint32_t>(std::atoi(env));
		if (b == 512 || b == 1024)
			runs_block_ = b;
	}
	use_runs_ = f32_ && S_ == 4 && runs_tile_ * C_ <= 512;
	// groups of 128 threads per tensor-core CTA (B3G_TC20_GROUPS = 1 or 2;
	// default: chosen per launch from the grid size)
	if (const char *env = std::getenv("B3G_TC20_CLUSTER")) {
		const int k = std::atoi(env);
		if (k >= 1 && k <= 8) {
			tc20_cluster_ = static_cast<uint32_t>(k);
			tc20_cluster_fixed_ = true;
		}
	}
	if (const char *env = std::getenv("B3G_TC20_GROUPS")) {
		const int gr = std::atoi(env);
		if (gr == 1 || gr == 2) {
			tc20_groups_ = static_cast<uint32_t>(gr);
			tc20_groups_fixed_ = true;
		}
	}
	// 20-state FP32 lists on the tensor cores: B3G_TC20=1, or a launch shape
	// of that engine fixed by one of the two switches above
	// (B3G_TC20=0: not at all, the autotuner does not try it either)
	use_tc20_ = f32_ && S_ == 20 && (tc20_cluster_fixed_ || tc20_groups_fixed_);
	bool tc20_off = false;
	if (const char *env = std::getenv("B3G_TC20")) {
		use_tc20_ = f32_ && S_ == 20 && std::atoi(env) != 0;
		tc20_off = std::atoi(env) == 0;
	}
	tc20_by_list_ = f32_ && S_ == 20 && !use_tc20_ && !tc20_off;
	// groups of the FP64 run form (B3G_F64_GROUPS: 1, 2, 4, 8 or 16 where
	// they fit a block; default: chosen per list)
	if (const char *env = std::getenv("B3G_F64_GROUPS")) {
		const int gr = std::atoi(env);
		if (gr == 1 || gr == 2 || gr == 4 || gr == 8 || gr == 16)
			f64_groups_ = static_cast<uint32_t>(gr);
	}
	if (const char *env = std::getenv("B3G_S20_GROUPS")) {
		const int gr = std::atoi(env);
		if (gr >= 1 && gr <= 4) {
			s20_groups_ = static_cast<uint32_t>(gr);
			tc20_by_list_ = false;
		}
	}
	// fused single-launch evaluation of short lists (B3G_DIRECT=0 turns
	// it off, e.g. to time the two-kernel path)
	use_direct_ = f32_ && S_ == 4 && (C_ == 1 || C_ == 2 || C_ == 4);
	if (const char *env = std::getenv("B3G_DIRECT"))
		use_direct_ = use_direct_ && std::atoi(env) != 0;

	use_tree_ = f32_ && S_ == 4 && C_ <= 16 && (uint64_t)C_ * ldp_ < (1ull << 28);
	// the switches of the run walk's form select the run walk
	for (const char *name : {"B3G_RUNS_TILE", "B3G_RUNS_BLOCK", "B3G_RUNS_SLOTS",
				 "B3G_RUNS_INLINE"})
		use_tree_ = use_tree_ && !std::getenv(name);
	if (const char *env = std::getenv("B3G_TREE"))
		use_tree_ = use_tree_ && std::atoi(env) != 0, tree_always_ = std::atoi(env) == 2;
	if (const char *env = std::getenv("B3G_TREE_GROUPS")) {
		const int gr = std::atoi(env);
		if (gr >= 1 && gr <= 16)
			tree_groups_ = static_cast<uint32_t>(gr);
	}
	if (use_tree_) { // the first list finds its workspaces
		tree_swap_.assign(I_, 0);
		list_ops_.resize(I_);
		for (auto *v : {&order_, &pos_of_, &tree_order_, &tree_ends_, &segs_})
			v->assign(I_ + 1, 0);
		nodes_.resize(I_ + 1);
		kid_.assign(2ull * I_, 0);
	}
	if (const char *env = std::getenv("B3G_TREE_TILE"))
		tree_tile_fixed_ = std::atoi(env) == 128 ? 128u : 64u;

	selectors_.assign(I_, 0);
	stamp_.assign(2 * L_ - 1, 0);
	pos_.assign(2 * L_ - 1, 0);
	run_of_.assign(I_, 0);
	smem_of_.assign(2ull * I_ + 1, static_cast<uint8_t>(kNoSlot));
	if (f32_ && S_ == 20)
		for (uint32_t w = 1; w <= 4; ++w)
			s20_per_sm_[w] = prune20_blocks_per_sm(w);
	// shared-memory slots of the run walk (B3G_RUNS_SLOTS=0: children of
	// listed entries read back from global memory, to time the difference)
	if (const char *env = std::getenv("B3G_RUNS_SLOTS"))
		use_slots_ = std::atoi(env) != 0;
	// per-run tables built by the run walk itself (B3G_RUNS_INLINE=0: a
	// separate transition kernel writes every table to global memory)
	if (const char *env = std::getenv("B3G_RUNS_INLINE"))
		use_inline_ = std::atoi(env) != 0;
	{
		int per_sm = 0, reserved = 0;
		check_cuda(cudaDeviceGetAttribute(
				   &per_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor,
				   device_),
			   "shared memory per SM");
		check_cuda(cudaDeviceGetAttribute(
				   &reserved, cudaDevAttrReservedSharedMemoryPerBlock,
				   device_),
			   "reserved shared memory");
		smem_per_sm_ = static_cast<uint32_t>(per_sm);
		smem_reserved_ = static_cast<uint32_t>(reserved);
	}

	const size_t slots = 2ull * I_;
	const size_t rsz = f32_ ? sizeof(float) : sizeof(double);
	// one block sum per thread block of any walk: at most one block per
	// 16 patterns (the smallest run-walk tile)
	const size_t nblocks = ldp_ / 16;
	block_sums_cap_ = static_cast<uint32_t>(nblocks);

	try {
		check_cuda(cudaStreamCreateWithFlags(&stream_,
						     cudaStreamNonBlocking),
			   "cudaStreamCreate");
		check_cuda(cudaEventCreateWithFlags(&ev_stage_free_,
						    cudaEventDisableTiming),
			   "cudaEventCreate");
		check_cuda(cudaEventCreateWithFlags(&ev_model_free_,
						    cudaEventDisableTiming),
			   "cudaEventCreate");
		check_cuda(cudaEventCreate(&ev_span0_), "cudaEventCreate");
		check_cuda(cudaEventCreate(&ev_span1_), "cudaEventCreate");
		for (auto &slot : ring_) {
			check_cuda(cudaEventCreate(&slot.k0), "cudaEventCreate");
			check_cuda(cudaEventCreate(&slot.kmid), "cudaEventCreate");
			check_cuda(cudaEventCreate(&slot.k1), "cudaEventCreate");
		}

		dev_alloc(d_tips_, (size_t)L_ * ldp_, "tips");
		dev_alloc(d_partials_, slots * C_ * ldp_ * S_ * rsz, "partials");
		dev_alloc(d_scales_, slots * C_ * ldp_ * sizeof(int32_t), "scales");
		dev_alloc(d_weights_, ldp_ * sizeof(uint32_t), "weights");
		dev_alloc(d_site_, ldp_ * sizeof(double), "site lnl");
		dev_alloc(d_cat_, (size_t)C_ * ldp_ * sizeof(double), "cat lnl");
		dev_alloc(d_block_sums_, nblocks * sizeof(double), "block sums");
		dev_alloc(d_ticket_, sizeof(unsigned), "ticket");
		dev_alloc(d_lnl_, sizeof(double), "lnl");
		if (f32_ && S_ == 20 && !tc20_off) {
			dev_alloc(d_tc_tab_, (size_t)I_ * 2 * C_ * 2 * 768 * sizeof(float),
				  "tensor-core tables");
			dev_alloc(d_status_, sizeof(unsigned), "status");
			check_cuda(cudaMemset(d_status_, 0, sizeof(unsigned)), "zero status");
			check_cuda(cudaHostAlloc((void **)&h_status_, sizeof(unsigned),
						 cudaHostAllocDefault),
				   "pinned status");
			*h_status_ = 0;
		}
		if (S_ == 20) {
			dev_alloc(d_root_val_, (size_t)C_ * ldp_ * sizeof(double), "root values");
			dev_alloc(d_root_exp_, (size_t)C_ * ldp_ * sizeof(int32_t), "root exponents");
			dev_alloc(d_tile_tickets_, ldp_ / 32 * sizeof(unsigned), "tile tickets");
			check_cuda(cudaMemset(d_tile_tickets_, 0, ldp_ / 32 * sizeof(unsigned)),
				   "zero tickets");
		}
		dev_alloc(d_model_, sizeof(ModelDev), "model");
		dev_alloc(d_ptab_, (size_t)I_ * 2 * C_ * (S_ + 1) * S_ * rsz,
			  "transition tables");
		if (!f32_ && S_ == 20)
			dev_alloc(d_soft20_, (size_t)I_ * 2 * C_ * soft_tab20_bytes(),
				  "integer transition tables");
		if (!f32_ && S_ == 4)
			dev_alloc(d_soft_, (size_t)I_ * 2 * C_ * sizeof(SoftTab4),
				  "integer transition tables");

		off_pi_ = align_up((size_t)I_ * sizeof(NodeOp), 256);
		off_runs_ = align_up(off_pi_ + S_ * sizeof(double), 256);
		off_slots_ = align_up(off_runs_ + (size_t)(I_ + 1) * sizeof(uint32_t), 256);
		off_tree_ = align_up(off_slots_ + (size_t)I_ * sizeof(uint32_t), 256);
		off_in_ = off_tree_;
		if (use_tree_)
			off_in_ = align_up(off_tree_ + (size_t)I_ * sizeof(TreeOp), 256);
		stage_bytes_ = off_in_ + (size_t)I_ * 2 * C_ * S_ * S_ * sizeof(double);
		dev_alloc(d_stage_, stage_bytes_, "stage");
		check_cuda(cudaHostAlloc((void **)&h_stage_, stage_bytes_,
					 cudaHostAllocDefault),
			   "pinned stage");
		check_cuda(cudaHostAlloc((void **)&h_model_, sizeof(ModelDev),
					 cudaHostAllocDefault),
			   "pinned model");
		// mapped: the fused short-list kernel writes the result here
		check_cuda(cudaHostAlloc((void **)&h_lnl_, sizeof(double),
					 cudaHostAllocMapped),
			   "pinned lnl");
		check_cuda(cudaHostGetDevicePointer((void **)&d_lnl_host_, h_lnl_, 0),
			   "mapped lnl");
		check_cuda(cudaHostAlloc((void **)&h_bsums_, block_sums_cap_ * sizeof(double),
					 cudaHostAllocMapped),
			   "pinned block sums");
		check_cuda(cudaHostGetDevicePointer((void **)&d_bsums_, h_bsums_, 0),
			   "mapped block sums");

		// DNA: single bases -> 0..3, everything else -> unknown (4)
		// (cpu4.rs:117-124).  Protein: states 0..19 as given, anything
		// else -> unknown (20).  Padded patterns are unknown too.
		std::vector<uint8_t> tips((size_t)L_ * ldp_, (uint8_t)S_);
		for (uint32_t l = 0; l < L_; ++l)
			for (uint32_t p = 0; p < P_; ++p) {
				const uint8_t code = samples[(size_t)l * P_ + p];
				uint8_t s;
				if (S_ == 4)
					s = code == 1 ? 0 : code == 2 ? 1
						   : code == 4 ? 2
						   : code == 8 ? 3
							       : 4;
				else
					s = code < S_ ? code : (uint8_t)S_;
				tips[(size_t)l * ldp_ + p] = s;
			}
		check_cuda(cudaMemcpy(d_tips_, tips.data(), tips.size(),
				      cudaMemcpyHostToDevice),
			   "upload tips");
		std::vector<uint32_t> w(ldp_, 0);
		for (uint32_t p = 0; p < P_; ++p)
			w[p] = 1;
		check_cuda(cudaMemcpy(d_weights_, w.data(), ldp_ * sizeof(uint32_t),
				      cudaMemcpyHostToDevice),
			   "upload weights");
		// Buffer::zeroed partials (cpu4.rs:134-136)
		check_cuda(cudaMemset(d_partials_, 0, slots * C_ * ldp_ * S_ * rsz),
			   "zero partials");
		check_cuda(cudaMemset(d_scales_, 0,
				      slots * C_ * ldp_ * sizeof(int32_t)),
			   "zero scales");
		check_cuda(cudaMemset(d_ticket_, 0, sizeof(unsigned)), "ticket");

		std::memset(&model_host_, 0, sizeof(model_host_));
		model_host_.states = S_;
		for (uint32_t c = 0; c < C_; ++c)
			model_host_.cat_rates[c] = 1.0;
		upload_model();
		check_cuda(cudaStreamSynchronize(stream_), "construct sync");
	} catch (...) {
		release();
		throw;
	}
}

Calculator::~Calculator() { release(); }

void Calculator::release()
{
	if (device_ >= 0)
		cudaSetDevice(device_);
	if (stream_)
		cudaStreamSynchronize(stream_);
	cudaFree(d_tips_);
	cudaFree(d_partials_);
	cudaFree(d_scales_);
	cudaFree(d_weights_);
	cudaFree(d_site_);
	cudaFree(d_cat_);
	cudaFree(d_tc_tab_);
	cudaFree(d_root_val_);
	cudaFree(d_root_exp_);
	cudaFree(d_status_);
	if (h_status_)
		cudaFreeHost(h_status_);
	d_tc_tab_ = nullptr;
	d_root_val_ = nullptr;
	d_root_exp_ = nullptr;
	d_status_ = nullptr;
	h_status_ = nullptr;
	cudaFree(d_block_sums_);
	cudaFree(d_ticket_);
	cudaFree(d_lnl_);
	cudaFree(d_model_);
	cudaFree(d_ptab_);
	cudaFree(d_soft_);
	d_soft_ = nullptr;
	cudaFree(d_soft20_);
	d_soft20_ = nullptr;
	cudaFree(d_tile_tickets_);
	d_tile_tickets_ = nullptr;
	cudaFree(own_d_stage_ ? own_d_stage_ : d_stage_);
	cudaFreeHost(own_h_stage_ ? own_h_stage_ : h_stage_);
	own_d_stage_ = nullptr;
	own_h_stage_ = nullptr;
	cudaFreeHost(h_model_);
	cudaFreeHost(h_lnl_);
	cudaFreeHost(h_bsums_);
	h_bsums_ = d_bsums_ = nullptr;
	d_tips_ = nullptr;
	d_partials_ = nullptr;
	d_scales_ = nullptr;
	d_weights_ = nullptr;
	d_site_ = d_cat_ = d_block_sums_ = d_lnl_ = nullptr;
	d_ticket_ = nullptr;
	d_model_ = nullptr;
	d_ptab_ = nullptr;
	d_stage_ = nullptr;
	h_stage_ = nullptr;
	h_model_ = nullptr;
	h_lnl_ = nullptr;
	for (cudaEvent_t *e : {&ev_stage_free_, &ev_model_free_, &ev_span0_,
			       &ev_span1_})
		if (*e) {
			cudaEventDestroy(*e);
			*e = nullptr;
		}
	for (auto &slot : ring_)
		for (cudaEvent_t *e : {&slot.k0, &slot.kmid, &slot.k1})
			if (*e) {
				cudaEventDestroy(*e);
				*e = nullptr;
			}
	if (stream_) {
		cudaStreamDestroy(stream_);
		stream_ = nullptr;
	}
}

void Calculator::upload_model()
{
	check_cuda(cudaEventSynchronize(ev_model_free_), "model staging");
	std::memcpy(h_model_, &model_host_, sizeof(ModelDev));
	check_cuda(cudaMemcpyAsync(d_model_, h_model_, sizeof(ModelDev),
				   cudaMemcpyHostToDevice, stream_),
		   "upload model");
	check_cuda(cudaEventRecord(ev_model_free_, stream_), "event");
	stream_dirty_ = true;
}

// The dirty list must name distinct internals, children must be valid node
// ids, and an internal child that is itself listed must come first
// (children-first order of partials_lists, parameters/tree.rs:398-421).
void Calculator::validate_lists(const uint32_t *internals,
				const uint32_t *children, uint32_t n)
{
	if (!internals || !children)
		throw Error(B3G_ERR_INVALID_ARGUMENT, "null list");
	if (n < 1 || n > I_)
		throw Error(B3G_ERR_INVALID_ARGUMENT,
			    "dirty list length must be in 1..num_internals");
	const uint32_t nodes = 2 * L_ - 1;
	// two stamps per call: `listed` marks the dirty internals, `done` the
	// ones already visited in list order
	if (stamp_epoch_ > 0xfffffff0u) {
		std::fill(stamp_.begin(), stamp_.end(), 0u);
		stamp_epoch_ = 0;
	}
	const uint32_t listed = ++stamp_epoch_;
	const uint32_t done = ++stamp_epoch_;
	for (uint32_t i = 0; i < n; ++i) {
		const uint32_t v = internals[i];
		if (v < L_ || v >= nodes)
			throw Error(B3G_ERR_INVALID_ARGUMENT,
				    "dirty list entry is not an internal node");
		if (stamp_[v] == listed)
			throw Error(B3G_ERR_INVALID_ARGUMENT,
				    "dirty list names a node twice");
		stamp_[v] = listed;
	}
	for (uint32_t i = 0; i < n; ++i) {
		const uint32_t v = internals[i];
		const uint32_t l = children[2 * i], r = children[2 * i + 1];
		for (const uint32_t ch : {l, r}) {
			if (ch >= nodes || ch == v)
				throw Error(B3G_ERR_INVALID_ARGUMENT,
					    "child is not a node id");
			if (ch >= L_ && stamp_[ch] == listed)
				throw Error(B3G_ERR_INVALID_ARGUMENT,
					    "dirty list is not children-first");
		}
		if (l == r)
			throw Error(B3G_ERR_INVALID_ARGUMENT,
				    "both children are the same node");
		stamp_[v] = done;
	}
}

namespace {
// c ? a : b without a branch.  Branches on a list's shape are mispredicted
// unless the same list comes again: with them the schedules of 32 whole trees of
// 184 taxa took 10.1 us each, more than the batch's depth-first kernel saved, now
// 5.5 (a step of such lists, 1,172 patterns x 4 categories: 566 us by the run
// walk, 643, 488); one tree over and over took 4.8 and takes 5.1.
uint32_t pick(bool c, uint32_t a, uint32_t b) { return b ^ ((a ^ b) & (0u - (uint32_t)c)); }

// At least n elements (growing again and again would clear them every time).
template <typename T> void fit(std::vector<T> &v, size_t n)
{
	if (v.size() < n)
		v.resize(n);
}
} // namespace

// Flips the selectors of the listed internals (Cpu4Calculator::
// set_selectors, cpu4.rs:93-98) and writes the schedule: output slot of each
// listed node and the slot or leaf of each child.
void Calculator::stage_ops(const uint32_t *internals, const uint32_t *children,
			   uint32_t n, bool tree)
{
	for (uint32_t i = 0; i < n; ++i)
		set_edited(selectors_[internals[i] - L_]);
	NodeOp *ops = reinterpret_cast<NodeOp *>(h_stage_);
	auto slot_of = [&](uint32_t v) {
		const uint32_t k = v - L_;
		return k * 2 + (selectors_[k] & 1u);
	};
	if (tree) {
		depth_first_ = order_depth_first(internals, children, n);
		if (depth_first_) {
			stage_tree(n);
			return;
		}
	}
	// Runs of mutually independent entries: entry i opens a new run when
	// one of its children is listed inside the current run.  validate_lists
	// left stamp_[v] == stamp_epoch_ on every listed internal.
	// A run holds at most kRunCap / C entries, so that the run walk's
	// per-run transition tables fit shared memory.
	uint32_t run_start = 0;
	const uint32_t cap = std::max(8u, kRunCap / C_);
	tip_children_ = 0;
	for (uint32_t i = 0; i < n; ++i) {
		if (i - run_start >= cap)
			run_start = i;
		NodeOp op;
		op.out = slot_of(internals[i]);
		const uint32_t l = children[2 * i], r = children[2 * i + 1];
		op.left = l < L_ ? (kTipBit | l) : slot_of(l);
		op.right = r < L_ ? (kTipBit | r) : slot_of(r);
		tip_children_ += (l < L_) + (r < L_);
		for (const uint32_t ch : {l, r})
			if (ch >= L_ && stamp_[ch] == stamp_epoch_ &&
			    pos_[ch] >= run_start)
				run_start = i;
		pos_[internals[i]] = i;
		run_of_[i] = run_start;
		ops[i] = op;
	}
	// NodeOp::pad = entries left in the run, this one included
	for (uint32_t i = n; i-- > 0;)
		ops[i].pad = (i + 1 < n && run_of_[i + 1] == run_of_[i])
				     ? ops[i + 1].pad + 1
				     : 1;
	// run starts, then n
	uint32_t *runs = reinterpret_cast<uint32_t *>(h_stage_ + off_runs_);
	n_runs_ = 0;
	max_run_ = 0;
	for (uint32_t i = 0; i < n; ++i)
		if (run_of_[i] == i) {
			if (n_runs_)
				max_run_ = std::max(max_run_, i - runs[n_runs_ - 1]);
			runs[n_runs_++] = i;
		}
	runs[n_runs_] = n;
	if (n_runs_)
		max_run_ = std::max(max_run_, n - runs[n_runs_ - 1]);
	if (tc20_by_list_)
		use_tc20_ = tc20_list(n);
	depth_first_ = S_ == 4 ? !f32_ : f32_ && !use_tc20_;
	if (!depth_first_)
		return;
	order_depth_first(internals, children, n);
	stage_order(n);
}

// Schedule of the depth-first FP32 walk (tree4.cuh) for the ordered list:
// group after group, child sources, and shared-memory slots for the outputs
// that the group's next entry does not take from registers and for the clean
// children.  Follows the kernel's order of events: before the first entry of
// chunk q the clean children of chunk q + 2 are copied; an entry's slots are
// read before its output is stored.  A slot returns to the group that read it
// (a slot that another group filled was read behind a barrier), so no other
// group can still be reading it when it is written again.  What finds no slot
// is read from global memory.
void Calculator::stage_tree(uint32_t n)
{
	const uint32_t G = order_groups_, phases = order_phases_;
	PruneParams pp{};
	pp.C = C_;
	pp.groups = G;
	pp.num_leaves = L_;
	const uint32_t tile = tree_tile_, budget = tree_budget(G);
	pp.tile = tile;
	pp.n_slots = 1;
	pp.tips_smem = 4ull * tip_children_ >= L_ &&
		       prune4_tree_smem(pp) + (size_t)tile * (L_ + 1) <= budget;
	TreeOp *ops = reinterpret_cast<TreeOp *>(h_stage_ + off_tree_);
	uint32_t *segs = reinterpret_cast<uint32_t *>(h_stage_ + off_runs_);
	TreeHead *heads = reinterpret_cast<TreeHead *>(segs + G + 1);
	// phase-major (order_, segs_) to group-major
	fit(tree_order_, n);
	fit(tree_ends_, (size_t)G * phases);
	uint32_t at = 0;
	for (uint32_t g = 0; g < G; ++g) {
		segs[g] = at;
		for (uint32_t ph = 0; ph < phases; ++ph) {
			for (uint32_t k = segs_[ph * G + g]; k < segs_[ph * G + g + 1]; ++k)
				tree_order_[at++] = order_[k];
			tree_ends_[ph * G + g] = at;
		}
	}
	segs[G] = n;
	order_.swap(tree_order_);
	// children's kinds: the group's previous output first, a tip last
	const NodeOp *const words = list_ops_.data();
	uint8_t *const swaps = tree_swap_.data();
	for (uint32_t g = 0; g < G; ++g) {
		uint32_t prev = kNone;
		for (uint32_t e = segs[g]; e < segs[g + 1]; ++e) {
			const NodeOp &in = words[order_[e]];
			const uint32_t l = in.left, r = in.right;
			const uint32_t swap = (uint32_t)(r == prev) |
					      ((uint32_t)(l != prev) & ((l & ~r) / kTipBit));
			const uint32_t flip = (l ^ r) & (0u - swap), a = l ^ flip, b = r ^ flip;
			const uint32_t code = (~a / kTipBit) * kTreeInA | (~b / kTipBit) * kTreeInB |
					      (uint32_t)(a == prev) * kTreePrev;
			swaps[e] = static_cast<uint8_t>(swap);
			ops[e] = TreeOp{in.out, code, 0, 0, {a, b}, 0, 0};
			prev = in.out;
		}
	}
	// (a whole tree's list has no child outside it)
	const bool any_clean = 2 * n - tip_children_ != n - 1;
	const uint32_t none = 2 * I_; // smem_of_ holds kNoSlot there
	uint32_t slots_used = 0;
	// (byte stores may alias the members)
	uint8_t *const smem = smem_of_.data();
	const uint32_t *const order = order_.data();
	auto assign = [&]() -> uint32_t { // entries and children without a slot
		const size_t rest = prune4_tree_smem(pp);
		const uint32_t capacity =
			1 + static_cast<uint32_t>(std::min<size_t>(
				    254, rest < budget ? (budget - rest) / (tile * 20 * C_) : 0));
		uint32_t used = 0, missing = 0, have[16] = {};
		uint8_t pool[16][258]; // a group's free slots: [1] .. [have]
		tree_clean_ = false;
		auto take = [&](const uint8_t *free, uint32_t &h, bool want) -> uint32_t {
			const bool old = want & (h != 0), fresh = want & !old & (used < capacity);
			const uint32_t s = pick(old, free[h], pick(fresh, used, kNoSlot));
			h -= old;
			used += fresh;
			missing += want & !old & !fresh;
			return s;
		};
		auto fetch = [&](uint32_t g, uint32_t chunk) { // its clean children
			const uint32_t lo = segs[g] + chunk * kTreeChunk;
			for (uint32_t e = lo; e < std::min(lo + kTreeChunk, segs[g + 1]); ++e) {
				const uint32_t *kid = &kid_[2 * (size_t)order[e]];
				for (uint32_t j = 0; j < 2; ++j) {
					if (!(ops[e].code & (j ? kTreeInB : kTreeInA)) ||
					    kid[j ^ tree_swap_[e]] != n)
						continue;
					const uint32_t s = take(pool[g], have[g], true);
					if (s == kNoSlot) {
						ops[e].code |= j ? kTreeMemB : kTreeMemA;
						continue;
					}
					ops[e].more |= (j ? kTreeCleanB : kTreeCleanA) |
						       s << (j ? 16 : 8);
					tree_clean_ = true;
				}
			}
		};
		for (auto &free : pool)
			free[0] = 0;
		for (uint32_t g = 0; any_clean && g < G; ++g) {
			fetch(g, 0);
			fetch(g, 1);
		}
		// a child that waits in a slot: its slot is free behind the entry
		auto read = [&](const TreeOp &op, uint32_t j, uint32_t &code, uint32_t &more,
				uint8_t *free, uint32_t &h) {
			const uint32_t mem = j ? kTreeMemB : kTreeMemA, shift = j ? 16 : 8;
			const bool need = ((code & (j ? kTreeInB : kTreeInA)) != 0) &
					  ((code & mem) == 0);
			const bool clean = more & (j ? kTreeCleanB : kTreeCleanA);
			const uint32_t kept = smem[pick(need & !clean, op.id[j], none)];
			const uint32_t s = pick(clean, more >> shift & 0xFFu, kept);
			if (need & (s == kNoSlot)) {
				code |= mem;
				return;
			}
			more |= pick(need & !clean, s << shift, 0u);
			free[h + 1] = static_cast<uint8_t>(s);
			h += need;
		};
		for (uint32_t ph = 0; ph < phases; ++ph)
			for (uint32_t g = 0; g < G; ++g) {
				uint8_t *const free = pool[g];
				uint32_t h = have[g];
				const uint32_t from = ph ? tree_ends_[(ph - 1) * G + g] : segs[g];
				const uint32_t to = tree_ends_[ph * G + g], end = segs[g + 1];
				for (uint32_t e = from; e < to; ++e) {
					if (any_clean && (e - segs[g]) % kTreeChunk == 0) {
						have[g] = h;
						fetch(g, (e - segs[g]) / kTreeChunk + 2);
						h = have[g];
					}
					TreeOp &op = ops[e];
					uint32_t code = op.code, more = op.more;
					// (rare but for clean children)
					if ((code & (kTreeInA | kTreePrev)) == kTreeInA)
						read(op, 0, code, more, free, h);
					read(op, 1, code, more, free, h);
					// the root, and what the next entry takes from registers,
					// need no slot
					const bool last = e + 1 == end;
					const bool keep = (order[e] != n - 1) &
							  (last | !(ops[e + !last].code & kTreePrev));
					const uint32_t s = take(free, h, keep);
					smem[op.out] = static_cast<uint8_t>(s);
					op.code = code | pick(s != kNoSlot, kTreeKeep | s << 8, 0u);
					op.more = more;
				}
				have[g] = h;
			}
		slots_used = used;
		return missing;
	};
	if (assign() && pp.tips_smem) { // the tips' room for slots
		pp.tips_smem = 0;
		for (uint32_t e = 0; e < n; ++e) {
			ops[e].code &= kTreeInA | kTreeInB | kTreePrev;
			ops[e].more = 0;
			smem_of_[ops[e].out] = static_cast<uint8_t>(kNoSlot);
		}
		(void)assign();
	}
	for (uint32_t i = 0; i < n; ++i)
		smem_of_[ops[i].out] = static_cast<uint8_t>(kNoSlot);
	tree_slots_ = std::max(1u, slots_used);
	tree_tips_ = pp.tips_smem;
	// what the words and heads read ahead, and the ends of the phases
	const uint32_t other = pp.tips_smem ? L_ * tile : kTreeNoTip;
	const uint32_t row = pp.tips_smem ? tile : 1u;
	auto tip = [&](uint32_t id) { return pick(id / kTipBit, (id & ~kTipBit) * row, other); };
	const uint32_t slot0 = prune4_tree_slot(G, tile, 0);
	const uint32_t pitch = prune4_tree_slot(G, tile, 1) - slot0;
	const uint32_t step = prune4_tree_entry(0, 1) - prune4_tree_entry(0, 0);
	for (uint32_t g = 0; g < G; ++g) {
		const uint32_t lo = segs[g], hi = segs[g + 1];
		TreeHead &h = heads[g];
		h = TreeHead{};
		const uint32_t entry0 = prune4_tree_entry(g, 0);
		TreeOp first[2] = {}; // stand for the two words before the group's first
		TreeOp *before = &first[0], *last = &first[1];
		for (uint32_t e = lo; e < hi; ++e) {
			TreeOp &op = ops[e];
			last->next_a = tip(op.id[0]);
			before->after_b = tip(op.id[1]);
			last->code |= pick(op.code & kTreeInB, slot0 + (op.more >> 16 & 0xFFu) * pitch,
					   entry0 + (e - lo) % kTreeRing * step)
				      << 16;
			before = last;
			last = &op;
		}
		h.tip[0] = first[1].next_a;
		h.tip[1] = first[0].after_b;
		h.tip[2] = first[1].after_b;
		h.base = first[1].code >> 16;
		// (the last phase needs no barrier)
		for (uint32_t ph = 0; ph + 1 < phases; ++ph) {
			const uint32_t end = tree_ends_[ph * G + g];
			if (end == lo) {
				++h.barriers;
			} else {
				ops[end - 1].code |= kTreeBarrier;
				++ops[end - 1].barriers;
			}
		}
	}
}

// Shared-memory slots for the run walk's outputs (at most `capacity`),
// written as per-entry codes beside the schedule.  A listed child is read
// by exactly one entry, its parent, so an entry may write its output into
// its left (else right) child's slot; an entry without a slotted child
// takes a slot released in an earlier run; the slot of a second slotted
// child is released at the end of the run.  Outputs left without a slot,
// and the last entry's, are read from global memory (or, for the last,
// from registers).  Returns the number of slots used.
uint32_t Calculator::assign_slots(uint32_t n, uint32_t capacity)
{
	if (capacity == 0)
		return 0;
	const NodeOp *ops = reinterpret_cast<const NodeOp *>(h_stage_);
	uint32_t *codes = reinterpret_cast<uint32_t *>(h_stage_ + off_slots_);
	free_slots_.clear();
	pending_slots_.clear();
	for (uint32_t k = capacity; k-- > 0;)
		free_slots_.push_back(static_cast<uint8_t>(k));
	auto src = [&](uint32_t id) -> uint32_t {
		return (id & kTipBit) ? kNoSlot : smem_of_[id];
	};
	uint32_t used = 0;
	for (uint32_t i = 0; i < n; ++i) {
		if (run_of_[i] == i) {
			free_slots_.insert(free_slots_.end(), pending_slots_.begin(),
					   pending_slots_.end());
			pending_slots_.clear();
		}
		const uint32_t ls = src(ops[i].left), rs = src(ops[i].right);
		uint32_t os = kNoSlot;
		if (i + 1 < n) {
			if (ls != kNoSlot) {
				os = ls;
				if (rs != kNoSlot)
					pending_slots_.push_back(static_cast<uint8_t>(rs));
			} else if (rs != kNoSlot) {
				os = rs;
			} else if (!free_slots_.empty()) {
				os = free_slots_.back();
				free_slots_.pop_back();
			}
		}
		smem_of_[ops[i].out] = static_cast<uint8_t>(os);
		if (os != kNoSlot)
			used = std::max(used, os + 1);
		codes[i] = os | (ls << 8) | (rs << 16);
	}
	for (uint32_t i = 0; i < n; ++i)
		smem_of_[ops[i].out] = static_cast<uint8_t>(kNoSlot);
	return used;
}

// Tile and groups of the depth-first FP32 walk.  128 patterns a block where
// there are more 64-pattern tiles than SMs (the table rows are read once for
// four columns instead of two), and groups until an SM has its warps (12, or
// 16 of the smaller tile) or the list's tips and slots fit the block's share
// of shared memory.  Us per whole tree at 64 / 128 patterns (4 categories):
// 256 taxa x 17,764 patterns 98 / 88, 128 x 30,000 94 / 84, 256 x 12,000 91 /
// 84; 256 x 8,000, 125 small tiles, 61 / 83, 64 x 7,855 34 / 37.  With 1 / 2 /
// 4 groups of the smaller tile: 256 x 8,000 94 / 72 / 62; of the larger: 256 x
// 17,764 118 / 88 / 91.
uint32_t Calculator::pick_tree(uint32_t n)
{
	PruneParams pp{};
	pp.C = C_;
	pp.num_leaves = L_;
	pp.tips_smem = 4ull * tip_children_ >= L_;
	uint32_t G = 1;
	if (tree_batch_) {
		tree_tile_ = 64;
		G = tree_groups_ ? tree_groups_ : std::max(1u, n / 8);
		return std::min(G, 16u / C_);
	}
	for (uint32_t tile = ldp_ / 64u > num_sms_ ? 128u : 64u;; tile = 64u) {
		if (tree_tile_fixed_)
			tile = tree_tile_fixed_;
		tree_tile_ = pp.tile = tile;
		const uint32_t blocks = ldp_ / tile, warps = tile == 128 ? 12 : 16;
		for (G = 1;; G *= 2) {
			if (tree_groups_)
				return tree_groups_ = std::min(tree_groups_, 16u / C_);
			const bool more = 2 * G * C_ <= 16 && 8 * G <= n;
			if (more && 2 * G * C_ * blocks <= warps * num_sms_)
				continue;
			pp.groups = G;
			pp.n_slots = 5 + 3 * G;
			if (prune4_tree_smem(pp) <= tree_budget(G))
				return G;
			if (!more)
				break;
		}
		if (tile == 64 || tree_tile_fixed_)
			return G;
	}
}

// Whether a batched list takes that walk: where its tips and slots fit a
// block.  Us a step, run walk / depth first, every member a whole tree of 4
// categories: 32 of 184 taxa x 1,172 patterns 276 / 183, 4 of 256 x 1,418 90 /
// 72, 8 of 64 x 857 46 / 39, 2 of 256 x 285 61 / 58; 2 of 700 x 300, too large,
// 114 / 132.
bool Calculator::batch_tree(uint32_t n) const
{
	PruneParams pp{};
	pp.C = C_;
	pp.num_leaves = L_;
	pp.tile = 64;
	pp.tips_smem = 1;
	pp.groups = std::min(std::max(1u, n / 8), 16u / C_);
	pp.n_slots = 3 + 5 * pp.groups / 2;
	return prune4_tree_smem(pp) <= kBatchTreeSmem;
}

// Shared memory of a block of that walk.
uint32_t Calculator::tree_budget(uint32_t G) const
{
	if (tree_batch_)
		return kBatchTreeSmem;
	const uint32_t warps = tree_tile_ == 128 ? 12 : 16;
	const uint32_t rounds = (ldp_ / tree_tile_ + num_sms_ - 1) / num_sms_;
	return smem_budget(1024u / std::max(1u, std::min(warps / (G * C_), rounds)));
}

// Groups a block of the depth-first walks (each walks subtrees of its own
// before one of them walks the entries above).
uint32_t Calculator::pick_groups(uint32_t n)
{
	if (S_ == 4 && f32_)
		return pick_tree(n);
	if (S_ == 20) {
		if (s20_groups_)
			return s20_groups_;
		// the most warps with which every block still runs at once: us
		// per whole tree with 1 / 2 / 3 / 4, 128 taxa x 4,989 patterns x 4
		// categories (624 blocks): 198 / 165 / 181 / 169; 61 x 2,003 x 4:
		// 89 / 73 / 70 / 67
		const uint32_t blocks = ldp_ / 32u * C_;
		uint32_t G = 1;
		for (uint32_t w = 2; w <= 4; ++w)
			if (4 * w <= n && s20_per_sm_[w] * num_sms_ >= blocks)
				G = w;
		return G;
	}
	if (f64_groups_)
		return C_ * f64_groups_ <= 16 ? f64_groups_ : 1u;
	// doubled while every block still runs at once (16 warps an SM at this
	// kernel's registers): us per whole tree with 1 / 2 / 4 / 8 groups, 37
	// taxa x 1,147 patterns: 51 / 41 / 35 / 36; 64 x 7,855, one category: 70 /
	// 54 / 48 / 50, four: 84 / 75 / 92; 128 x 17,764, one category: 130 / 99 /
	// 80 / 93
	const uint32_t warps = ldp_ / 32u * C_;
	uint32_t G = 1;
	while (2 * G * C_ <= 16 && 8 * G <= n && 2 * G * warps <= 16 * num_sms_)
		G *= 2;
	return G;
}

// Whether the walk of G groups holds the phases (the 20-state FP32 and the
// four-state FP64 walk keep them in shared memory).
bool Calculator::segs_fit(uint32_t G) const
{
	return S_ == 20 ? segs_.size() <= prune20_seg_words(G)
			: f32_ || segs_.size() <= prune4_f64_seg_words(G * C_);
}

// The phases of G groups (segs_, and pos_of_ the entries above and the pieces'
// roots); false where they would not
// shorten the longest group's work by a fifth.
bool Calculator::split_phases(uint32_t n, uint32_t G)
{
	above_mark_.assign(n, 0);
	uint32_t at = 0;
	// split the costliest subtree until the pieces balance; what is split
	// belongs to the entries above
	std::vector<uint32_t> &piece = pieces_, &above = above_;
	piece.assign(1, n - 1);
	above.clear();
	while (!piece.empty() && piece.size() < 4 * G) {
		uint64_t most = 0; // the first of the costliest
		for (size_t k = 0; k < piece.size(); ++k)
			most = std::max(most, (uint64_t)nodes_[piece[k]].cost << 32 | (uint32_t)~k);
		const size_t top = (uint32_t)~(uint32_t)most;
		const uint32_t v = piece[top];
		if (v != n - 1 && nodes_[v].cost * 2 * G <= nodes_[n - 1].cost)
			break;
		above.push_back(v);
		above_mark_[v] = 1;
		piece[top] = piece.back();
		piece.pop_back();
		for (int j = 0; j < 2; ++j)
			if (kid_[2 * v + j] != n)
				piece.push_back(kid_[2 * v + j]);
	}
	std::sort(piece.begin(), piece.end(), [&](uint32_t a, uint32_t b) {
		return nodes_[a].cost != nodes_[b].cost ? nodes_[a].cost > nodes_[b].cost : a < b;
	});
	std::sort(above.begin(), above.end()); // children first
	// a piece goes to the least loaded group
	uint32_t load[16] = {}, owner[80];
	for (size_t k = 0; k < piece.size(); ++k) {
		owner[k] = (uint32_t)(std::min_element(load, load + G) - load);
		load[owner[k]] += nodes_[piece[k]].cost;
	}
	segs_.clear();
	for (uint32_t w = 0; w < G; ++w) {
		segs_.push_back(at);
		for (size_t k = 0; k < piece.size(); ++k)
			if (owner[k] == w) {
				at += nodes_[piece[k]].size;
				pos_of_[piece[k]] = at - 1;
			}
	}
	uint32_t longest = *std::max_element(load, load + G);
	// the entries above: runs of independent entries, each dealt out in
	// contiguous shares
	uint32_t phases = 1;
	for (size_t i = 0; i < above.size();) {
		size_t j = i;
		for (; j < above.size(); ++j) {
			bool free = true;
			for (size_t k = i; k < j; ++k)
				free = free && kid_[2 * above[j]] != above[k] &&
				       kid_[2 * above[j] + 1] != above[k];
			if (!free)
				break;
		}
		const uint32_t len = (uint32_t)(j - i);
		for (uint32_t w = 0; w < G; ++w) {
			segs_.push_back(at + (len * w + G - 1) / G);
		}
		for (size_t k = i; k < j; ++k)
			pos_of_[above[k]] = at++;
		longest += (len + G - 1) / G * 6 + 4; // entries, and the barrier
		++phases;
		i = j;
	}
	segs_.push_back(at);
	if (longest * 5 > nodes_[n - 1].cost * 4 || segs_.size() > (size_t)I_ + 1) {
		segs_.assign({0u, n});
		return false;
	}
	order_groups_ = G;
	order_phases_ = phases;
	return true;
}

// The list's words (list_ops_), ordered depth first, heavier subtree first, so
// that a child is mostly the previous entry's output, and for several groups
// split into phases (segs_): disjoint subtrees, a balanced share a group, then
// the entries above them, run by run.  Every entry's arithmetic is the same
// in any children-first order.  order_[k] = list position of staged entry k.
// A list that is not one tree under its last entry keeps its order (false).
bool Calculator::order_depth_first(const uint32_t *internals, const uint32_t *children,
				   uint32_t n)
{
	fit(order_, n);
	fit(list_ops_, n);
	fit(kid_, 2 * (size_t)n);
	fit(pos_of_, (size_t)n + 1);
	fit(nodes_, (size_t)n + 1);
	// (in locals: the stores below could alias the members)
	const uint32_t *const stamp = stamp_.data();
	const uint8_t *const sel = selectors_.data();
	uint32_t *const pos = pos_.data(), *const kids = kid_.data();
	ListNode *const nodes = nodes_.data();
	NodeOp *const words = list_ops_.data();
	const uint32_t L = L_, epoch = stamp_epoch_;
	// a child that is not listed is entry n, of cost and size zero
	nodes[n] = ListNode{0, 0, 0, kNone};
	uint32_t linked = 0, inner = 0, twice = 0;
	for (uint32_t i = 0; i < n; ++i) {
		// an entry's cost: 2, and 3 more for each internal child
		uint32_t cost = 2, size = 1, chain = 0, id[2], ins = 0;
		for (int j = 0; j < 2; ++j) {
			const uint32_t v = children[2 * i + j];
			const uint32_t in = v < L ? 0u : kNone; // masks
			const uint32_t k = (v - L) & in;
			id[j] = ((kTipBit | v) & ~in) | ((2 * k + (sel[k] & 1u)) & in);
			ins += in & 1u;
			// (validate_lists left stamp_epoch_ on every listed internal)
			const uint32_t is = stamp[v] == epoch ? kNone : 0u;
			const uint32_t at = n + ((pos[v] - n) & is);
			ListNode &kid = nodes[at];
			twice |= (kid.parent + 1u) & is;
			kid.parent = i;
			kids[2 * i + j] = at;
			cost += kid.cost;
			size += kid.size;
			chain = std::max(chain, kid.chain);
			linked += is & 1u;
		}
		const uint32_t v = internals[i], k = v - L;
		words[i] = NodeOp{2 * k + (sel[k] & 1u), id[0], id[1], 0};
		pos[v] = i;
		inner += ins;
		nodes[i] = ListNode{cost + 3 * ins, chain + 2 + 3 * ins, size, kNone};
	}
	const bool tree = twice == 0;
	tip_children_ = 2 * n - inner;
	order_groups_ = 1;
	order_phases_ = 1;
	segs_.assign({0u, n});
	if (!tree || linked + 1 != n) {
		for (uint32_t i = 0; i < n; ++i)
			order_[i] = i;
		return false;
	}
	// at most twice the list's work over its longest chain
	uint32_t G = pick_groups(n);
	while (G > 1 && G * nodes_[n - 1].chain > 2 * nodes_[n - 1].cost)
		G = S_ == 20 ? G - 1 : G / 2;
	bool split = G > 1 && split_phases(n, G);
	// a long ladder's phases may be too many: fewer groups hold more
	while (split && !segs_fit(G)) {
		G = S_ == 20 ? G - 1 : G / 2;
		split = G > 1 && split_phases(n, G);
	}
	if (!split) {
		order_groups_ = order_phases_ = 1;
		segs_.assign({0u, n});
		above_mark_.assign(n, 0);
		pos_of_[n - 1] = n - 1;
	}
	// post-order from the roots' places down, the heavier child's subtree
	// first, so that the lighter child ends just before its parent
	uint32_t *const place = pos_of_.data(), *const order = order_.data();
	const uint8_t *const above = above_mark_.data();
	for (uint32_t v = n; v-- > 0;) {
		const uint32_t at = place[v];
		order[at] = v;
		const uint32_t a = kids[2 * v], b = kids[2 * v + 1];
		const uint32_t flip = (a ^ b) & (0u - (uint32_t)(nodes[a].cost < nodes[b].cost));
		const uint32_t heavy = a ^ flip, light = b ^ flip;
		// (the children of an entry above the pieces have their places)
		const uint32_t set = above[v] - 1u;
		place[n + ((light - n) & set)] = at - 1;
		place[n + ((heavy - n) & set)] = at - 1 - nodes[light].size;
	}
	return true;
}

// The ordered list's schedule words (the walks but the FP32 four-state one).
void Calculator::stage_order(uint32_t n)
{
	NodeOp *ops = reinterpret_cast<NodeOp *>(h_stage_);
	size_t seg = 0; // segs_[seg]: where the current walk began
	for (uint32_t k = 0; k < n; ++k) {
		NodeOp op = list_ops_[order_[k]];
		bool first = false; // of its walk
		for (; seg < segs_.size() && segs_[seg] <= k; ++seg)
			first = first || segs_[seg] == k;
		const uint32_t prev = first ? kNone : ops[k - 1].out;
		const bool lp = op.left == prev, rp = op.right == prev;
		const bool lt = (op.left & kTipBit) != 0, rt = (op.right & kTipBit) != 0;
		// first the child that is not the previous output; of the others a
		// partial before a tip
		op.pad = lp ? kS20Swap | kS20Prev : rp ? kS20Prev : lt && !rt ? kS20Swap : 0u;
		ops[k] = op;
	}
	if (order_groups_ > 1)
		std::memcpy(h_stage_ + off_runs_, segs_.data(), segs_.size() * sizeof(uint32_t));
}

// The list's edge lengths (two values an entry) or matrices into the staging
// block, in the staged order.
void Calculator::stage_inputs(const double *src, uint32_t n, size_t per_entry)
{
	double *dst = reinterpret_cast<double *>(h_stage_ + off_in_);
	if (!depth_first_) {
		std::memcpy(dst, src, n * per_entry * sizeof(double));
		return;
	}
	if (S_ == 4 && f32_) { // children in the schedule's order
		const size_t half = per_entry / 2;
		for (uint32_t k = 0; half == 1 && k < n; ++k) { // lengths
			dst[2 * k] = src[2 * order_[k] + tree_swap_[k]];
			dst[2 * k + 1] = src[2 * order_[k] + (tree_swap_[k] ^ 1u)];
		}
		if (half == 1)
			return;
		for (uint32_t k = 0; k < n; ++k)
			for (uint32_t j = 0; j < 2; ++j)
				std::memcpy(dst + k * per_entry + j * half,
					    src + order_[k] * per_entry + (j ^ tree_swap_[k]) * half,
					    half * sizeof(double));
		return;
	}
	for (uint32_t k = 0; k < n; ++k)
		std::memcpy(dst + k * per_entry, src + order_[k] * per_entry,
			    per_entry * sizeof(double));
}

// Groups a block of the 20-state FP64 walk: doubled while a group's share of
// a run stays at two thirds of an entry and at most four groups share an SM
// (us per whole tree with 1 / 2 / 4 groups: 61 taxa x 2,003 patterns x 4
// categories 378 / 301 / 276, one category 359 / 285 / 261; 64 x 2,500 x 4,
// 160 blocks: 512 / 489 / 515; 128 x 4,989 x 4, 312 blocks: the same).
uint32_t Calculator::pick_p20_groups(uint32_t n) const
{
	if (f64_groups_)
		return std::min(f64_groups_, 4u);
	const uint32_t blocks = ldp_ / 64u * C_;
	uint32_t G = 1;
	while (G < 4 && 4 * G * n_runs_ <= 3 * n && 2 * G * blocks <= 4 * num_sms_)
		G *= 2;
	return G;
}

void Calculator::launch(uint32_t n, bool matrices_mode, double clock_rate,
			bool want_cat)
{
	host_fold_blocks_ = 0;
	if (use_direct_ && !matrices_mode && !want_cat && n > 0 &&
	    n <= kDirectMax) {
		launch_direct(n, clock_rate);
		return;
	}
	// run walk configuration, decided before the upload because the slot
	// codes travel with the schedule
	const bool tree = S_ == 4 && f32_ && depth_first_;
	const bool runs = S_ == 4 && use_runs_ && n <= 4096 && !tree;
	PruneParams pp{};
	uint32_t block = 512;
	if (runs) {
		pp.n = n;
		pp.C = C_;
		pp.num_leaves = L_;
		pp.n_runs = n_runs_;
		pp.tile = pick_tile(n);
		pp.tips_smem = (4ull * tip_children_ >= L_ &&
				(size_t)L_ * pp.tile <= 32u * 1024u)
				       ? 1u
				       : 0u;
		pp.ptab_smem = (size_t)n * 2 * C_ * 5 * 16 <= kPtabSmemBytes ? 1u : 0u;
		const uint32_t cols = pp.tile * C_;
		// 1024-thread blocks only for the run walk proper (a 512-column
		// tile is the serial walk of a 512-thread block)
		block = (runs_block_ == 1024 && cols < 512) ? 1024u : 512u;
		const uint32_t budget = smem_budget(block);
		if (use_inline_ && block / cols >= 2 && max_run_ > 0) {
			// the walk builds each run's tables itself, one run ahead
			pp.tables_inline = 1;
			pp.ptab_smem = 0;
			pp.max_run = max_run_;
			pp.lengths_smem = (!matrices_mode && n <= 1024) ? 1u : 0u;
			if (prune4_runs_smem(pp) > budget) {
				pp.tables_inline = 0;
				pp.max_run = 0;
				pp.lengths_smem = 0;
				pp.ptab_smem = (size_t)n * 2 * C_ * 5 * 16 <= kPtabSmemBytes
						       ? 1u
						       : 0u;
			}
		}
		if (use_slots_ && block / cols >= 2) {
			// as many slots as fit beside the rest
			pp.n_slots = 1;
			const size_t one = prune4_runs_smem(pp);
			const size_t per = (size_t)cols * (sizeof(float4) + sizeof(int32_t));
			const size_t cap = one <= budget ? 1 + (budget - one) / per : 0;
			pp.n_slots = assign_slots(
				n, static_cast<uint32_t>(std::min<size_t>(cap, kNoSlot - 1)));
		}
	}
	const size_t in_bytes =
		matrices_mode ? (size_t)n * 2 * C_ * S_ * S_ * sizeof(double)
			      : (size_t)n * 2 * sizeof(double);
	// (the depth-first FP32 walk's schedule lies behind the list's)
	const size_t from = tree ? off_pi_ : 0;
	last_upload_bytes_ = off_in_ + in_bytes - from;
	check_cuda(cudaMemcpyAsync(d_stage_ + from, h_stage_ + from, last_upload_bytes_,
				   cudaMemcpyHostToDevice, stream_),
		   "upload step");
	check_cuda(cudaEventRecord(ev_stage_free_, stream_), "event");
	upload_pending_ = true;
	TimingSlot &slot = ring_[ring_next_ % kRing];
	if (slot.pending)
		harvest(slot); // recorded kRing proposals ago: long complete
	slot.direct = false;
	record(slot.k0);

	if (S_ == 20) {
		launch20(n, matrices_mode, clock_rate, want_cat, slot);
		return;
	}
	PtabParams pt{};
	pt.lengths = matrices_mode
			     ? nullptr
			     : reinterpret_cast<const double *>(d_stage_ + off_in_);
	pt.matrices = matrices_mode
			      ? reinterpret_cast<const double *>(d_stage_ + off_in_)
			      : nullptr;
	pt.model = d_model_;
	pt.clock_rate = clock_rate;
	pt.n = n;
	pt.C = C_;
	pt.ptab = d_ptab_;
	pt.soft = d_soft_;
	if (pp.tables_inline) {
		pp.model = d_model_;
		pp.lengths = pt.lengths;
		pp.matrices = pt.matrices;
		pp.clock_rate = clock_rate;
		last_launches_ = 1;
	} else {
		check_cuda(tree ? launch_ptab4_rows(pt, stream_) : launch_ptab4(pt, f32_, stream_),
			   "transition kernel");
		last_launches_ = 2;
	}
	record(slot.kmid);

	pp.tips = d_tips_;
	pp.partials = d_partials_;
	pp.scales = d_scales_;
	pp.ops = reinterpret_cast<const NodeOp *>(d_stage_);
	pp.ptab = d_ptab_;
	pp.soft = d_soft_;
	pp.pi = reinterpret_cast<const double *>(d_stage_ + off_pi_);
	pp.weights = d_weights_;
	pp.site_lnl = d_site_;
	pp.cat_lnl = want_cat ? d_cat_ : nullptr;
	pp.block_sums = d_block_sums_;
	pp.ticket = d_ticket_;
	pp.lnl_out = d_lnl_;
	pp.n = n;
	pp.ldp = ldp_;
	pp.C = C_;
	pp.scale_ln = scale_ln_;
	pp.num_leaves = L_;
	// stage the tip tile when the list reads at least a quarter of the
	// leaves and the tile fits in 64 KiB of shared memory (the run walk
	// decided its own above)
	if (!runs)
		pp.tips_smem = (4ull * tip_children_ >= L_ &&
				(size_t)L_ * tile_ <= 64u * 1024u)
				       ? 1u
				       : 0u;
	pp.scale_threshold = std::exp(-static_cast<double>(scale_ln_));
	pp.scale_mult = std::exp(static_cast<double>(scale_ln_));
	std::copy(scale_pow_, scale_pow_ + kScalePow, pp.scale_pow);
	pp.log_inv_c = std::log(1.0 / static_cast<double>(C_));
	// the run-synchronous walk stages the schedule in shared memory: keep
	// it for lists up to 4,096 entries
	if (tree) {
		pp.ops = reinterpret_cast<const NodeOp *>(d_stage_ + off_tree_);
		pp.n_slots = tree_slots_;
		pp.tips_smem = tree_tips_;
		pp.groups = order_groups_;
		pp.phases = order_phases_;
		pp.segs = reinterpret_cast<const uint32_t *>(d_stage_ + off_runs_);
		pp.sums_host = d_bsums_;
		arm_host_fold(ldp_ / tree_tile_);
		pp.tile = tree_tile_;
		check_cuda(launch_prune4_tree(pp, tree_clean_, stream_), "pruning kernel");
	} else if (runs) {
		pp.runs = reinterpret_cast<const uint32_t *>(d_stage_ + off_runs_);
		pp.slots = reinterpret_cast<const uint32_t *>(d_stage_ + off_slots_);
		const uint32_t tiles = ldp_ / pp.tile;
		const uint32_t ctas = std::min(tiles, num_sms_ * (1024 / block));
		if (ctas > block_sums_cap_)
			throw Error(B3G_ERR_STATE, "run walk grid exceeds the block sums");
		// the blocks' sums go straight to mapped host memory
		if (d_bsums_) {
			pp.sums_host = d_bsums_;
			arm_host_fold(ctas);
		} else {
			pp.lnl_host = d_lnl_host_;
			arm_poll();
		}
		check_cuda(launch_prune4_runs(pp, ctas, block, stream_), "pruning kernel");
	} else {
		poll_result_ = false;
		if (pp.soft) { // the blocks' sums go to mapped host memory here too
			pp.groups = order_groups_;
			pp.phases = order_phases_;
			pp.segs = reinterpret_cast<const uint32_t *>(d_stage_ + off_runs_);
			pp.sums_host = d_bsums_;
			arm_host_fold(ldp_ / (pp.groups > 1 ? 32u : tile_));
		}
		check_cuda(launch_prune4(pp, f32_, tile_, stream_), "pruning kernel");
	}
	++in_flight_;
	record(slot.k1);
	slot.pending = timing_;
	ring_next_ += timing_ ? 1 : 0;
	if (!pp.sums_host && !pp.lnl_host)
		check_cuda(cudaMemcpyAsync(h_lnl_, d_lnl_, sizeof(double),
					   cudaMemcpyDeviceToHost, stream_),
			   "read lnl");
	have_result_ = true;
	outstanding_ = true;
	stream_dirty_ = true;
	cat_valid_ = want_cat;
}

// 20-state list: table kernel, then the column walk (prune20.cuh).
void Calculator::launch20(uint32_t n, bool matrices_mode, double clock_rate,
			  bool want_cat, TimingSlot &slot)
{
	poll_result_ = false; // (the tcgen05 walk's result is read back by a copy)
	PtabParams pt{};
	pt.lengths = matrices_mode
			     ? nullptr
			     : reinterpret_cast<const double *>(d_stage_ + off_in_);
	pt.matrices = matrices_mode
			      ? reinterpret_cast<const double *>(d_stage_ + off_in_)
			      : nullptr;
	pt.model = d_model_;
	pt.clock_rate = clock_rate;
	pt.n = n;
	pt.C = C_;
	pt.ptab = d_ptab_;
	if (use_tc20_) {
		check_cuda(launch_ptab20tc(pt, d_tc_tab_, stream_), "transition kernel");
		last_launches_ = 3; // tables, pruning, root and sum
		record(slot.kmid);
		Tc20Params tp{};
		tp.tips = d_tips_;
		tp.partials = static_cast<float *>(d_partials_);
		tp.scales = d_scales_;
		tp.ops = reinterpret_cast<const NodeOp *>(d_stage_);
		tp.tab = static_cast<const float *>(d_ptab_);
		tp.tc_tab = d_tc_tab_;
		tp.pi = reinterpret_cast<const double *>(d_stage_ + off_pi_);
		tp.weights = d_weights_;
		tp.root_val = d_root_val_;
		tp.root_exp = d_root_exp_;
		tp.site_lnl = d_site_;
		tp.cat_lnl = want_cat ? d_cat_ : nullptr;
		tp.block_sums = d_block_sums_;
		tp.ticket = d_ticket_;
		tp.lnl_out = d_lnl_;
		tp.status = d_status_;
		tp.n = n;
		tp.ldp = ldp_;
		tp.C = C_;
		tp.L = L_;
		// the list, then the tile's tip codes, in shared memory when they
		// fit beside the operand areas at 4 / groups CTAs per SM
		// two groups (on independent entries of a run) unless the grid
		// holds six or more CTAs per SM, where one group per CTA and up to
		// four CTAs per SM hide the per-entry latency as well (measured:
		// two groups faster at 1 and 4.1 CTAs per SM, one at 10.2)
		const uint32_t groups =
			tc20_groups_ ? tc20_groups_
				     : ((ldp_ / 128u) * C_ < 6u * num_sms_ ? 2u : 1u);
		tp.groups = groups;
		// a work item (tile, category) spread over a cluster of CTAs
		// while the grid has fewer items than CTA slots (4 / groups per
		// SM), so that every SM holds groups on independent entries
		const uint32_t items = (ldp_ / 128u) * C_;
		uint32_t cluster = std::max(1u, std::min(8u, (4u / groups) * num_sms_ /
								      std::max(items, 1u)));
		if (tc20_cluster_fixed_)
			cluster = tc20_cluster_;
		tp.cluster = cluster;
		const size_t budget = smem_budget(256u * groups);
		const size_t ops_bytes = (size_t)n * sizeof(NodeOp);
		size_t used = prune20tc_smem(groups, false, n, false, L_);
		tp.ops_smem = used + ops_bytes <= budget ? 1u : 0u;
		used += tp.ops_smem ? ops_bytes : 0;
		tp.tips_smem = used + (size_t)L_ * 128u <= budget ? 1u : 0u;
		tp.log_inv_c = std::log(1.0 / static_cast<double>(C_));
		check_cuda(launch_prune20tc(tp, stream_), "tensor-core pruning kernel");
		++in_flight_;
		record(slot.k1);
		slot.pending = timing_;
		ring_next_ += timing_ ? 1 : 0;
		check_cuda(cudaMemcpyAsync(h_lnl_, d_lnl_, sizeof(double),
					   cudaMemcpyDeviceToHost, stream_),
			   "read lnl");
		check_cuda(cudaMemcpyAsync(h_status_, d_status_, sizeof(unsigned),
					   cudaMemcpyDeviceToHost, stream_),
			   "read status");
		have_result_ = true;
		outstanding_ = true;
		stream_dirty_ = true;
		cat_valid_ = want_cat;
		return;
	}
	pt.soft20 = d_soft20_;
	check_cuda(launch_ptab20(pt, f32_, stream_), "transition kernel");
	last_launches_ = 2;
	record(slot.kmid);
	PruneParams pp{};
	pp.tips = d_tips_;
	pp.partials = d_partials_;
	pp.scales = d_scales_;
	pp.ops = reinterpret_cast<const NodeOp *>(d_stage_);
	pp.ptab = d_ptab_;
	pp.pi = reinterpret_cast<const double *>(d_stage_ + off_pi_);
	pp.weights = d_weights_;
	pp.site_lnl = d_site_;
	pp.cat_lnl = want_cat ? d_cat_ : nullptr;
	pp.block_sums = d_block_sums_;
	pp.ticket = d_ticket_;
	pp.lnl_out = d_lnl_;
	pp.n = n;
	pp.ldp = ldp_;
	pp.C = C_;
	pp.scale_ln = scale_ln_;
	pp.num_leaves = L_;
	pp.scale_threshold = std::exp(-static_cast<double>(scale_ln_));
	pp.scale_mult = std::exp(static_cast<double>(scale_ln_));
	std::copy(scale_pow_, scale_pow_ + kScalePow, pp.scale_pow);
	pp.log_inv_c = std::log(1.0 / static_cast<double>(C_));
	pp.root_val = d_root_val_;
	pp.root_exp = d_root_exp_;
	pp.ticket = d_tile_tickets_;
	pp.runs = reinterpret_cast<const uint32_t *>(d_stage_ + off_runs_);
	pp.n_runs = n_runs_;
	pp.sums_host = d_bsums_;
	if (f32_) {
		pp.groups = order_groups_;
		pp.phases = order_phases_;
		pp.segs = pp.runs;
		arm_host_fold(ldp_ / 32u);
		check_cuda(launch_prune20(pp, stream_), "pruning kernel");
	} else {
		pp.soft20 = d_soft20_;
		arm_host_fold(ldp_ / 64u);
		check_cuda(launch_prune20_f64(pp, pick_p20_groups(n), stream_), "pruning kernel");
	}
	++in_flight_;
	record(slot.k1);
	slot.pending = timing_;
	ring_next_ += timing_ ? 1 : 0;
	have_result_ = true;
	outstanding_ = true;
	stream_dirty_ = true;
	cat_valid_ = want_cat;
}

// One launch for a short FP32 list: the staged schedule, the lengths and
// the root frequencies go into the kernel parameters (nothing is uploaded),
// the kernel builds its transition tables in shared memory and writes the
// result into the mapped pinned word that log_likelihood() reads.
void Calculator::launch_direct(uint32_t n, double clock_rate)
{
	DirectParams dp;
	dp.tips = d_tips_;
	dp.partials = d_partials_;
	dp.scales = d_scales_;
	dp.weights = d_weights_;
	dp.model = d_model_;
	dp.site_lnl = d_site_;
	dp.block_sums = d_block_sums_;
	dp.ticket = d_ticket_;
	dp.lnl_out = d_lnl_;
	dp.lnl_host = d_lnl_host_;
	dp.sums_host = d_bsums_;
	dp.n = n;
	dp.ldp = ldp_;
	dp.L = L_;
	dp.C = C_;
	dp.clock_rate = clock_rate;
	dp.log_inv_c = std::log(1.0 / static_cast<double>(C_));
	std::memcpy(dp.pi, h_stage_ + off_pi_, 4 * sizeof(double));
	for (int k = 0; k < 16; ++k) {
		dp.eig[k] = static_cast<float>(model_host_.V[k]);
		dp.eig[16 + k] = static_cast<float>(model_host_.Vinv[k]);
	}
	for (int k = 0; k < 4; ++k) {
		dp.eig[32 + k] = static_cast<float>(model_host_.lambda[k]);
		dp.rate[k] = clock_rate * model_host_.cat_rates[k];
	}
	dp.eig[36] = model_host_.shortcuts ? 1.0f : 0.0f;
	dp.eig[37] = dp.eig[38] = dp.eig[39] = 0.0f;
	std::memcpy(dp.ops, h_stage_, (size_t)n * sizeof(NodeOp));
	std::memcpy(dp.lengths, h_stage_ + off_in_, (size_t)n * 2 * sizeof(double));
	// where each child comes from in the walk
	for (uint32_t i = 0; i < n; ++i) {
		const uint32_t ids[2] = {dp.ops[i].left, dp.ops[i].right};
		uint32_t marks = 0;
		for (int j = 0; j < 2; ++j) {
			const uint32_t id = ids[j];
			uint32_t src = kSrcClean;
			if (id & kTipBit) {
				src = kSrcTip;
			} else if (i >= 1 && id == dp.ops[i - 1].out) {
				src = kSrcPrev;
			} else if (i >= 2 && id == dp.ops[i - 2].out) {
				src = kSrcPrev2;
			} else {
				for (uint32_t k = 0; k + 2 < i; ++k)
					if (dp.ops[k].out == id) {
						src = kSrcEarlier;
						break;
					}
			}
			marks |= src << (8 * j);
		}
		dp.ops[i].pad = marks;
	}
	// bytes that reach the device with the launch
	last_upload_bytes_ = (uint64_t)n * (sizeof(NodeOp) + 2 * sizeof(double)) +
			     4 * sizeof(double);
	TimingSlot &slot = ring_[ring_next_ % kRing];
	if (slot.pending)
		harvest(slot);
	slot.direct = true;
	record(slot.k0);
	// 128-pattern tiles, 128 * C threads per block, 1024 threads per SM
	const uint32_t ctas = std::min(ldp_ / 128u, (8u / C_) * num_sms_);
	if (ctas > block_sums_cap_)
		throw Error(B3G_ERR_STATE, "short-list grid exceeds the block sums");
	if (d_bsums_)
		arm_host_fold(ctas);
	else
		arm_poll();
	check_cuda(launch_prune4_direct(dp, ctas, stream_), "fused pruning kernel");
	++in_flight_;
	last_launches_ = 1;
	record(slot.k1);
	slot.pending = timing_;
	ring_next_ += timing_ ? 1 : 0;
	have_result_ = true;
	outstanding_ = true;
	stream_dirty_ = true;
	cat_valid_ = false;
}

void Calculator::propose_matrices(const uint32_t *internals,
				  const uint32_t *children, uint32_t n,
				  const double *matrices, const double *freqs)
{
	DeviceGuard g(device_);
	validate_lists(internals, children, n);
	if (!matrices || !freqs)
		throw Error(B3G_ERR_INVALID_ARGUMENT, "null matrices");
	if (own_h_stage_)
		throw Error(B3G_ERR_STATE,
			    "a calculator in a batch takes edge-length proposals only");
	const size_t count = (size_t)n * 2 * C_ * S_ * S_;
	for (size_t k = 0; k < count; ++k)
		if (!std::isfinite(matrices[k]))
			throw Error(B3G_ERR_NUMERIC, "non-finite transition matrix");
	for (uint32_t s = 0; s < S_; ++s)
		if (!std::isfinite(freqs[s]))
			throw Error(B3G_ERR_NUMERIC, "non-finite frequency");
	wait_stage();
	stage_ops(internals, children, n, tree_list(n));
	std::memcpy(h_stage_ + off_pi_, freqs, S_ * sizeof(double));
	stage_inputs(matrices, n, 2ull * C_ * S_ * S_);
	launch(n, true, 1.0, true);
}

void Calculator::propose_lengths(const uint32_t *internals,
				 const uint32_t *children, uint32_t n,
				 const double *lengths, double clock_rate)
{
	DeviceGuard g(device_);
	if (!model_set_)
		throw Error(B3G_ERR_STATE,
			    "no substitution model set before propose_lengths");
	validate_lists(internals, children, n);
	if (!lengths)
		throw Error(B3G_ERR_INVALID_ARGUMENT, "null lengths");
	for (size_t k = 0; k < (size_t)n * 2; ++k)
		if (!std::isfinite(lengths[k]))
			throw Error(B3G_ERR_NUMERIC, "non-finite edge length");
	if (!std::isfinite(clock_rate))
		throw Error(B3G_ERR_NUMERIC, "non-finite clock rate");
	wait_stage();
	wait_batch();
	stage_ops(internals, children, n,
		  tree_list(n) && !(use_direct_ && n <= kDirectMax));
	std::memcpy(h_stage_ + off_pi_, model_host_.pi, S_ * sizeof(double));
	stage_inputs(lengths, n, 2);
	staged_ = false;
	launch(n, false, clock_rate, false);
}

void Calculator::stage_lengths(const uint32_t *internals,
			       const uint32_t *children, uint32_t n,
			       const double *lengths, double clock_rate)
{
	DeviceGuard g(device_);
	if (!in_batch_)
		throw Error(B3G_ERR_STATE,
			    "stage_lengths needs the calculator to be in a batch");
	if (!model_set_)
		throw Error(B3G_ERR_STATE,
			    "no substitution model set before stage_lengths");
	if (n > 4096)
		throw Error(B3G_ERR_INVALID_ARGUMENT,
			    "batched lists hold at most 4,096 entries");
	validate_lists(internals, children, n);
	if (!lengths)
		throw Error(B3G_ERR_INVALID_ARGUMENT, "null lengths");
	for (size_t k = 0; k < (size_t)n * 2; ++k)
		if (!std::isfinite(lengths[k]))
			throw Error(B3G_ERR_NUMERIC, "non-finite edge length");
	if (!std::isfinite(clock_rate))
		throw Error(B3G_ERR_NUMERIC, "non-finite clock rate");
	// the batch's previous copy of this staging buffer must be done, and
	// so must this calculator's own last launch
	wait_stage();
	wait_batch();
	// (a batch takes short lists by one launch whatever B3G_DIRECT says)
	const bool is_short = n <= kDirectMax && (C_ == 1 || C_ == 2 || C_ == 4);
	tree_batch_ = true;
	stage_ops(internals, children, n, !is_short && use_tree_ && batch_tree(n));
	tree_batch_ = false;
	staged_kind_ = is_short ? kListShort : depth_first_ ? kListTree : kListRuns;
	std::memcpy(h_stage_ + off_pi_, model_host_.pi, S_ * sizeof(double));
	stage_inputs(lengths, n, 2);
	staged_ = true;
	staged_n_ = n;
	staged_clock_ = clock_rate;
	staged_tile_ = pick_tile(n);
	staged_tips_smem_ = (4ull * tip_children_ >= L_ &&
			     (size_t)L_ * staged_tile_ <= 32u * 1024u)
				    ? 1u
				    : 0u;
	have_result_ = false; // results come from the batch
}

void Calculator::likelihoods(double *out)
{
	DeviceGuard g(device_);
	if (!out)
		throw Error(B3G_ERR_INVALID_ARGUMENT, "null output");
	if (!have_result_ || !cat_valid_)
		throw Error(B3G_ERR_STATE,
			    "likelihoods() needs a preceding propose()");
	check_cuda(cudaMemcpy2DAsync(out, P_ * sizeof(double), d_cat_,
				     ldp_ * sizeof(double), P_ * sizeof(double),
				     C_, cudaMemcpyDeviceToHost, stream_),
		   "read likelihoods");
	check_cuda(cudaStreamSynchronize(stream_), "sync");
	upload_pending_ = false;
	in_flight_ = 0;
}

namespace {
// a NaN payload the kernels never write
constexpr uint64_t kLnlSentinel = 0x7ff4b3a9c0de5e11ull;
} // namespace

void Calculator::arm_poll()
{
	poll_result_ = in_flight_ == 0;
	if (poll_result_)
		std::memcpy(h_lnl_, &kLnlSentinel, sizeof(double));
}

void Calculator::arm_host_fold(uint32_t blocks)
{
	host_fold_blocks_ = blocks;
	poll_result_ = in_flight_ == 0;
	if (poll_result_)
		for (uint32_t k = 0; k < blocks; ++k)
			std::memcpy(h_bsums_ + k, &kLnlSentinel, sizeof(double));
}

// Waits for every block's mapped sum to leave the sentinel (the same
// stream queries as wait_mapped); false: the stream finished with a sum
// missing, or polling was not armed.
bool Calculator::wait_host_sums()
{
	const volatile uint64_t *w = reinterpret_cast<const volatile uint64_t *>(h_bsums_);
	uint32_t k = 0;
	for (uint32_t poll = 1; k < host_fold_blocks_; ++poll) {
		if (w[k] != kLnlSentinel) {
			++k;
			continue;
		}
		if ((poll & 63u) == 0) {
			const cudaError_t e = cudaStreamQuery(stream_);
			if (e == cudaSuccess) {
				for (; k < host_fold_blocks_; ++k)
					if (w[k] == kLnlSentinel)
						return false;
				return true;
			}
			if (e != cudaErrorNotReady)
				check_cuda(e, "evaluation");
		}
	}
	return true;
}

double Calculator::fold_host_sums() const
{
	return f32_ ? fold_block_sums(h_bsums_, host_fold_blocks_)
		    : fold_block_sums_compensated(h_bsums_, host_fold_blocks_);
}

// Waits for the mapped result word to leave the sentinel; every 64 polls
// the stream is queried, so a launch error surfaces and a stream that
// finished without writing the word ends the wait (false: synchronise).
bool Calculator::wait_mapped(double &value)
{
	const volatile uint64_t *w = reinterpret_cast<const volatile uint64_t *>(h_lnl_);
	for (uint32_t k = 1;; ++k) {
		uint64_t bits = *w;
		if (bits != kLnlSentinel) {
			std::memcpy(&value, &bits, sizeof(double));
			return true;
		}
		if ((k & 63u) == 0) {
			const cudaError_t e = cudaStreamQuery(stream_);
			if (e == cudaSuccess) {
				bits = *w;
				if (bits == kLnlSentinel)
					return false;
				std::memcpy(&value, &bits, sizeof(double));
				return true;
			}
			if (e != cudaErrorNotReady)
				check_cuda(e, "evaluation");
		}
	}
}

double Calculator::log_likelihood()
{
	DeviceGuard g(device_);
	if (!have_result_)
		throw Error(B3G_ERR_STATE, "no proposal evaluated yet");
	double value;
	if (host_fold_blocks_) {
		if (!(poll_result_ && wait_host_sums()))
			check_cuda(cudaStreamSynchronize(stream_), "sync");
		upload_pending_ = false;
		in_flight_ = 0;
		for (uint32_t k = 0; k < host_fold_blocks_; ++k) {
			uint64_t bits;
			std::memcpy(&bits, h_bsums_ + k, sizeof(bits));
			if (poll_result_ && bits == kLnlSentinel)
				throw Error(B3G_ERR_CUDA,
					    "the evaluation finished without writing its result");
		}
		value = fold_host_sums();
		// later reads return the folded value
		*h_lnl_ = value;
		host_fold_blocks_ = 0;
		poll_result_ = false;
		return value;
	}
	if (poll_result_ && wait_mapped(value)) {
		// the kernel ran, so the upload before it did too
		upload_pending_ = false;
		in_flight_ = 0;
		return value;
	}
	check_cuda(cudaStreamSynchronize(stream_), "sync");
	upload_pending_ = false;
	in_flight_ = 0;
	if (poll_result_) {
		uint64_t bits;
		std::memcpy(&bits, h_lnl_, sizeof(bits));
		if (bits == kLnlSentinel)
			throw Error(B3G_ERR_CUDA,
				    "the evaluation finished without writing its result");
	}
	if (h_status_ && *h_status_)
		throw Error(B3G_ERR_TIMEOUT,
			    "a tensor-core wait of the 20-state kernel gave up");
	return *h_lnl_;
}

void Calculator::site_log_likelihoods(double *out)
{
	DeviceGuard g(device_);
	if (!out)
		throw Error(B3G_ERR_INVALID_ARGUMENT, "null output");
	if (!have_result_)
		throw Error(B3G_ERR_STATE, "no proposal evaluated yet");
	check_cuda(cudaMemcpyAsync(out, d_site_, P_ * sizeof(double),
				   cudaMemcpyDeviceToHost, stream_),
		   "read site lnl");
	check_cuda(cudaStreamSynchronize(stream_), "sync");
	upload_pending_ = false;
	in_flight_ = 0;
}

// The staging buffer may be rewritten once the last upload from it has
// run: wait for that upload, unless the stream was synchronised since it
// was queued (the common case: the result was read before the next
// proposal).
void Calculator::wait_stage()
{
	if (upload_pending_) {
		check_cuda(cudaEventSynchronize(ev_stage_free_), "stage reuse");
		upload_pending_ = false;
	}
}

// A replay of the batch may still read this calculator's slice of the
// staging block, until its results have been read (Batch::log_likelihoods).
void Calculator::wait_batch()
{
	if (batch_done_ && batch_running_) {
		check_cuda(cudaEventSynchronize(batch_done_), "batch stage reuse");
		batch_running_ = false;
	}
}

void Calculator::record(cudaEvent_t e)
{
	if (timing_)
		check_cuda(cudaEventRecord(e, stream_), "event");
}

void Calculator::harvest(TimingSlot &s)
{
	check_cuda(cudaEventSynchronize(s.k1), "timing sync");
	float t = 0.0f, p = 0.0f;
	if (s.direct) { // one fused kernel: all of it counts as pruning
		check_cuda(cudaEventElapsedTime(&p, s.k0, s.k1), "elapsed");
	} else {
		check_cuda(cudaEventElapsedTime(&t, s.k0, s.kmid), "elapsed");
		check_cuda(cudaEventElapsedTime(&p, s.kmid, s.k1), "elapsed");
	}
	acc_transition_ms_ += t;
	acc_prune_ms_ += p;
	++acc_count_;
	s.pending = false;
}

void Calculator::last_timing(float *transition_ms, float *prune_ms)
{
	DeviceGuard g(device_);
	if (!timing_)
		throw Error(B3G_ERR_STATE,
			    "timing is off (b3g_calculator_set_timing)");
	if (!have_result_ || ring_next_ == 0)
		throw Error(B3G_ERR_STATE, "no proposal evaluated yet");
	TimingSlot &s = ring_[(ring_next_ - 1) % kRing];
	check_cuda(cudaEventSynchronize(s.k1), "sync");
	if (s.direct) {
		*transition_ms = 0.0f;
		check_cuda(cudaEventElapsedTime(prune_ms, s.k0, s.k1), "elapsed");
		return;
	}
	check_cuda(cudaEventElapsedTime(transition_ms, s.k0, s.kmid), "elapsed");
	check_cuda(cudaEventElapsedTime(prune_ms, s.kmid, s.k1), "elapsed");
}

void Calculator::timing_totals(bool reset, double *transition_ms,
			       double *prune_ms, uint64_t *proposals)
{
	DeviceGuard g(device_);
	// harvest in recording order
	const uint64_t first = ring_next_ > kRing ? ring_next_ - kRing : 0;
	for (uint64_t i = first; i < ring_next_; ++i) {
		TimingSlot &s = ring_[i % kRing];
		if (s.pending)
			harvest(s);
	}
	*transition_ms = acc_transition_ms_;
	*prune_ms = acc_prune_ms_;
	*proposals = acc_count_;
	if (reset) {
		acc_transition_ms_ = acc_prune_ms_ = 0.0;
		acc_count_ = 0;
	}
}

void Calculator::span_begin()
{
	DeviceGuard g(device_);
	check_cuda(cudaEventRecord(ev_span0_, stream_), "event");
}

float Calculator::span_end()
{
	DeviceGuard g(device_);
	check_cuda(cudaEventRecord(ev_span1_, stream_), "event");
	check_cuda(cudaEventSynchronize(ev_span1_), "sync");
	float ms = 0.0f;
	check_cuda(cudaEventElapsedTime(&ms, ev_span0_, ev_span1_), "elapsed");
	return ms;
}

uint32_t Calculator::autotune(const uint32_t *internals,
			      const uint32_t *children, uint32_t n,
			      const double *lengths, double clock_rate)
{
	DeviceGuard g(device_);
	if (!f32_)
		return 0;
	const bool timing = timing_;
	timing_ = true; // the trials read the kernel timings
	struct Restore {
		bool &flag;
		bool value;
		~Restore() { flag = value; }
	} restore{timing_, timing};
	// best of three timed evaluations after one warm-up, each rejected
	auto trial = [&]() {
		float best = INFINITY;
		for (int r = 0; r < 4; ++r) {
			propose_lengths(internals, children, n, lengths, clock_rate);
			(void)log_likelihood();
			float t = 0.0f, p = 0.0f;
			last_timing(&t, &p);
			reject();
			if (r > 0)
				best = std::min(best, t + p);
		}
		return best;
	};
	if (S_ == 20) {
		if (!d_tc_tab_) // built without tensor-core buffers
			return 0;
		tc20_by_list_ = false; // one choice for every list from here
		// tensor cores with one and with two thread groups per CTA
		// (unless B3G_TC20_GROUPS fixed it), then the register walk
		use_tc20_ = true;
		float tc = INFINITY;
		uint32_t best_groups = tc20_groups_;
		for (const uint32_t gr : {1u, 2u}) {
			if (tc20_groups_fixed_ && gr != tc20_groups_)
				continue;
			tc20_groups_ = gr;
			const float t = trial();
			if (t < tc) {
				tc = t;
				best_groups = gr;
			}
		}
		tc20_groups_ = best_groups;
		use_tc20_ = false;
		const float cc = trial();
		use_tc20_ = tc <= cc;
		return use_tc20_ ? 1u : 0u;
	}
	// the direct launch of short lists and path-like lists do not use the
	// tuned tile
	if (!use_runs_ || (use_direct_ && n <= kDirectMax))
		return runs_tile_;
	// (patterns per tile, threads per block).  Two pattern columns of one
	// category per thread: a warp spans 32 / (tile / 2) categories, so
	// tiles of 16 and 32 patterns put four and two categories in a warp
	// (and give small alignments more blocks), 64 and 128 one.
	// (The run walk's shape, for batches and lists of several trees; the
	// depth-first walk has none.)
	const bool tree = tree_list(n);
	Restore walk{use_tree_, use_tree_};
	use_tree_ = false;
	uint32_t best_tile = runs_tile_, best_block = runs_block_;
	float best_ms = INFINITY;
	const uint32_t cand[][2] = {{16, 512},  {32, 512},  {64, 512},
				    {128, 512}, {32, 1024}, {64, 1024}};
	for (const auto &tb : cand) {
		const uint32_t t = tb[0], b = tb[1];
		if (t * C_ > 512 || (b == 1024 && t * C_ >= 512))
			continue;
		runs_tile_ = t;
		runs_block_ = b;
		const float ms = trial();
		if (ms < best_ms) {
			best_ms = ms;
			best_tile = t;
			best_block = b;
		}
	}
	runs_tile_ = best_tile;
	runs_block_ = best_block;
	use_tree_ = walk.value;
	if (tree) // leave the walk that the list takes in the caches
		(void)trial();
	return best_tile;
}

void Calculator::accept()
{
	outstanding_ = false;
	// Cpu4Calculator::accept (cpu4.rs:78-83): EditBuf::accept
	for (auto &m : selectors_)
		m &= 1u;
}

void Calculator::reject()
{
	outstanding_ = false;
	// Cpu4Calculator::reject (cpu4.rs:85-89): EditBuf::reject
	for (auto &m : selectors_)
		m = static_cast<uint8_t>((m ^ (m >> 1)) & 1u);
}

void Calculator::set_weights(const uint32_t *w)
{
	DeviceGuard g(device_);
	if (!w)
		throw Error(B3G_ERR_INVALID_ARGUMENT, "null weights");
	std::vector<uint32_t> padded(ldp_, 0);
	std::memcpy(padded.data(), w, P_ * sizeof(uint32_t));
	check_cuda(cudaStreamSynchronize(stream_), "sync");
	upload_pending_ = false;
	in_flight_ = 0;
	check_cuda(cudaMemcpy(d_weights_, padded.data(), ldp_ * sizeof(uint32_t),
			      cudaMemcpyHostToDevice),
		   "upload weights");
}

void Calculator::set_eigen(const double *V, const double *Vinv,
			   const double *lambda, const double *Q,
			   const double *pi, int shortcuts)
{
	DeviceGuard g(device_);
	if (!V || !Vinv || !lambda || !Q || !pi)
		throw Error(B3G_ERR_INVALID_ARGUMENT, "null eigensystem");
	const uint32_t nn = S_ * S_;
	for (uint32_t k = 0; k < nn; ++k)
		if (!std::isfinite(V[k]) || !std::isfinite(Vinv[k]) ||
		    !std::isfinite(Q[k]))
			throw Error(B3G_ERR_NUMERIC, "non-finite eigensystem");
	for (uint32_t k = 0; k < S_; ++k)
		if (!std::isfinite(lambda[k]) || !std::isfinite(pi[k]))
			throw Error(B3G_ERR_NUMERIC, "non-finite eigensystem");
	std::memcpy(model_host_.V, V, nn * sizeof(double));
	std::memcpy(model_host_.Vinv, Vinv, nn * sizeof(double));
	std::memcpy(model_host_.Q, Q, nn * sizeof(double));
	std::memcpy(model_host_.lambda, lambda, S_ * sizeof(double));
	std::memcpy(model_host_.pi, pi, S_ * sizeof(double));
	model_host_.shortcuts = shortcuts ? 1u : 0u;
	upload_model();
	model_set_ = true;
}

void Calculator::set_reversible(const double *rates, const double *pi,
				int shortcuts)
{
	DeviceGuard g(device_);
	if (!rates || !pi)
		throw Error(B3G_ERR_INVALID_ARGUMENT, "null model");
	const uint32_t nr = S_ * (S_ - 1) / 2;
	double psum = 0.0;
	for (uint32_t k = 0; k < nr; ++k)
		if (!std::isfinite(rates[k]) || rates[k] < 0.0)
			throw Error(B3G_ERR_NUMERIC,
				    "exchangeabilities must be finite and >= 0");
	for (uint32_t k = 0; k < S_; ++k) {
		if (!std::isfinite(pi[k]) || !(pi[k] > 0.0))
			throw Error(B3G_ERR_NUMERIC,
				    "frequencies must be finite and > 0");
		psum += pi[k];
	}
	(void)psum;
	// decomposed on the host in FP64: a one-block Jacobi kernel measured
	// about 410 us per model on this GPU (its FP64 pipe issues at 1/64 of
	// the FP32 rate), the host takes a few microseconds
	const int sweeps = reversible_eigen((int)S_, rates, pi, model_host_.V,
					    model_host_.Vinv, model_host_.lambda,
					    model_host_.Q);
	if (sweeps < 0)
		throw Error(B3G_ERR_NUMERIC,
			    "eigen decomposition of Q did not converge");
	std::memcpy(model_host_.pi, pi, S_ * sizeof(double));
	model_host_.shortcuts = shortcuts ? 1u : 0u;
	upload_model();
	model_set_ = true;
}

void Calculator::set_category_rates(const double *rates)
{
	DeviceGuard g(device_);
	if (!rates)
		throw Error(B3G_ERR_INVALID_ARGUMENT, "null rates");
	for (uint32_t c = 0; c < C_; ++c)
		if (!std::isfinite(rates[c]) || rates[c] < 0.0)
			throw Error(B3G_ERR_NUMERIC, "bad category rate");
	// update only the category rates of the device model in place
	std::memcpy(model_host_.cat_rates, rates, C_ * sizeof(double));
	check_cuda(cudaEventSynchronize(ev_model_free_), "model staging");
	std::memcpy(h_model_->cat_rates, rates, C_ * sizeof(double));
	check_cuda(cudaMemcpyAsync(d_model_->cat_rates, h_model_->cat_rates,
				   C_ * sizeof(double), cudaMemcpyHostToDevice,
				   stream_),
		   "upload category rates");
	check_cuda(cudaEventRecord(ev_model_free_, stream_), "event");
	stream_dirty_ = true;
}

void Calculator::set_gamma(double alpha)
{
	if (!std::isfinite(alpha) || !(alpha > 0.0))
		throw Error(B3G_ERR_NUMERIC, "alpha must be finite and > 0");
	std::vector<double> r(C_);
	gamma_categories(alpha, static_cast<int>(C_), r.data());
	set_category_rates(r.data());
}

} // namespace b3g

// ===========================================================================
// C ABI

namespace {

thread_local std::string g_last_error;

template <typename F> b3g_status guarded(F &&f)
{
	try {
		f();
		g_last_error.clear();
		return B3G_OK;
	} catch (const b3g::Error &e) {
		g_last_error = e.what();
		return e.status;
	} catch (const std::bad_alloc &) {
		g_last_error = "host allocation failed";
		return B3G_ERR_OUT_OF_MEMORY;
	} catch (const std::exception &e) {
		g_last_error = e.what();
		return B3G_ERR_STATE;
	} catch (...) {
		g_last_error = "unknown error";
		return B3G_ERR_STATE;
	}
}

b3g::Calculator *calc_of(b3g_calculator *c)
{
	if (!c)
		throw b3g::Error(B3G_ERR_INVALID_ARGUMENT, "null calculator");
	return reinterpret_cast<b3g::Calculator *>(c);
}

} // namespace

namespace b3g {

// Records the outcome of an entry point defined in another translation unit
// in the per-thread message that b3g_last_error() returns.
void set_last_error(const char *message)
{
	g_last_error = message ? message : "";
}

} // namespace b3g

extern "C" {

B3G_API const char *b3g_last_error(void) { return g_last_error.c_str(); }

B3G_API const char *b3g_version(void) { return "b3g 0.1.0 sm_103a"; }

B3G_API b3g_status b3g_calculator_create(const b3g_config *config,
					 const uint8_t *samples,
					 b3g_calculator **out)
{
	return guarded([&] {
		if (!config || !out)
			throw b3g::Error(B3G_ERR_INVALID_ARGUMENT, "null argument");
		*out = nullptr;
		auto *c = new b3g::Calculator(*config, samples);
		*out = reinterpret_cast<b3g_calculator *>(c);
	});
}

B3G_API void b3g_calculator_destroy(b3g_calculator *calc)
{
	delete reinterpret_cast<b3g::Calculator *>(calc);
}

B3G_API uint32_t b3g_calculator_num_patterns(const b3g_calculator *calc)
{
	return calc ? reinterpret_cast<const b3g::Calculator *>(calc)->num_patterns()
		    : 0u;
}

B3G_API b3g_status b3g_calculator_propose(b3g_calculator *calc,
					  const uint32_t *internals,
					  const uint32_t *children, uint32_t n,
					  const double *matrices,
					  const double *frequencies)
{
	return guarded([&] {
		calc_of(calc)->propose_matrices(internals, children, n, matrices,
						frequencies);
	});
}

B3G_API b3g_status b3g_calculator_likelihoods(b3g_calculator *calc,
					      double *out)
{
	return guarded([&] { calc_of(calc)->likelihoods(out); });
}

B3G_API b3g_status b3g_calculator_accept(b3g_calculator *calc)
{
	return guarded([&] { calc_of(calc)->accept(); });
}

B3G_API b3g_status b3g_calculator_reject(b3g_calculator *calc)
{
	return guarded([&] { calc_of(calc)->reject(); });
}

B3G_API b3g_status b3g_calculator_set_weights(b3g_calculator *calc,
					      const uint32_t *weights)
{
	return guarded([&] { calc_of(calc)->set_weights(weights); });
}

B3G_API b3g_status b3g_calculator_set_eigen(b3g_calculator *calc,
					    const double *V,
					    const double *Vinv,
					    const double *lambda,
					    const double *Q,
					    const double *frequencies,
					    int shortcuts)
{
	return guarded([&] {
		calc_of(calc)->set_eigen(V, Vinv, lambda, Q, frequencies,
					 shortcuts);
	});
}

B3G_API b3g_status b3g_calculator_set_reversible(b3g_calculator *calc,
						 const double *rates,
						 const double *frequencies,
						 int shortcuts)
{
	return guarded([&] {
		calc_of(calc)->set_reversible(rates, frequencies, shortcuts);
	});
}

B3G_API b3g_status b3g_calculator_set_category_rates(b3g_calculator *calc,
						     const double *rates)
{
	return guarded([&] { calc_of(calc)->set_category_rates(rates); });
}

B3G_API b3g_status b3g_calculator_set_gamma(b3g_calculator *calc,
					    double alpha)
{
	return guarded([&] { calc_of(calc)->set_gamma(alpha); });
}

B3G_API b3g_status b3g_calculator_propose_lengths(b3g_calculator *calc,
						  const uint32_t *internals,
						  const uint32_t *children,
						  uint32_t n,
						  const double *lengths,
						  double clock_rate)
{
	return guarded([&] {
		calc_of(calc)->propose_lengths(internals, children, n, lengths,
					       clock_rate);
	});
}

B3G_API b3g_status b3g_calculator_log_likelihood(b3g_calculator *calc,
						 double *out)
{
	return guarded([&] {
		if (!out)
			throw b3g::Error(B3G_ERR_INVALID_ARGUMENT, "null output");
		*out = calc_of(calc)->log_likelihood();
	});
}

B3G_API b3g_status b3g_calculator_site_log_likelihoods(b3g_calculator *calc,
						       double *out)
{
	return guarded([&] { calc_of(calc)->site_log_likelihoods(out); });
}

B3G_API b3g_status b3g_calculator_set_timing(b3g_calculator *calc, int on)
{
	return guarded([&] { calc_of(calc)->set_timing(on != 0); });
}

B3G_API b3g_status b3g_calculator_last_timing(b3g_calculator *calc,
					      float *transition_ms,
					      float *prune_ms)
{
	return guarded([&] {
		if (!transition_ms || !prune_ms)
			throw b3g::Error(B3G_ERR_INVALID_ARGUMENT, "null output");
		calc_of(calc)->last_timing(transition_ms, prune_ms);
	});
}

B3G_API b3g_status b3g_calculator_timing_totals(b3g_calculator *calc,
						int reset,
						double *transition_ms,
						double *prune_ms,
						uint64_t *proposals)
{
	return guarded([&] {
		if (!transition_ms || !prune_ms || !proposals)
			throw b3g::Error(B3G_ERR_INVALID_ARGUMENT, "null output");
		calc_of(calc)->timing_totals(reset != 0, transition_ms, prune_ms,
					     proposals);
	});
}

B3G_API b3g_status b3g_calculator_last_upload_bytes(b3g_calculator *calc,
						    uint64_t *bytes)
{
	return guarded([&] {
		if (!bytes)
			throw b3g::Error(B3G_ERR_INVALID_ARGUMENT, "null output");
		*bytes = calc_of(calc)->last_upload_bytes();
	});
}

B3G_API b3g_status b3g_calculator_last_launches(b3g_calculator *calc,
						uint32_t *kernels)
{
	return guarded([&] {
		if (!kernels)
			throw b3g::Error(B3G_ERR_INVALID_ARGUMENT, "null output");
		*kernels = calc_of(calc)->last_launches();
	});
}

B3G_API b3g_status b3g_calculator_span_begin(b3g_calculator *calc)
{
	return guarded([&] { calc_of(calc)->span_begin(); });
}

B3G_API b3g_status b3g_calculator_span_end(b3g_calculator *calc, float *ms)
{
	return guarded([&] {
		if (!ms)
			throw b3g::Error(B3G_ERR_INVALID_ARGUMENT, "null output");
		*ms = calc_of(calc)->span_end();
	});
}

B3G_API b3g_status b3g_calculator_autotune(b3g_calculator *calc,
					   const uint32_t *internals,
					   const uint32_t *children, uint32_t n,
					   const double *lengths,
					   double clock_rate, uint32_t *choice)
{
	return guarded([&] {
		if (!choice)
			throw b3g::Error(B3G_ERR_INVALID_ARGUMENT, "null output");
		*choice = calc_of(calc)->autotune(internals, children, n, lengths,
						  clock_rate);
	});
}

} // extern "C"
