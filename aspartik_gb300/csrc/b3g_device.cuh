// b3g_device.cuh -- device-side layouts shared by the b3g kernels and the
// host orchestration.
//
// Device store of one calculator (one chain), all resident in HBM:
//   tips      u8  [L][ldp]                   state 0..S-1, S = unknown
//   partials  R   [2I][C][ldp][S]            slot = (v - L) * 2 + selector
//                                            (20 states, FP32: [10][128][2]
//                                            in each 128-pattern tile)
//   scales    i32 [2I][C][ldp]               cumulative rescale count of the
//                                            subtree below the slot's node
//   ptab      R   [n][2][C][S+1][S]          per-step transposed transition
//                                            tables, row S = all ones
// ldp is the pattern count rounded up to a multiple of 128; padded patterns
// carry unknown tips and weight 0.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "index_width.hpp"
#include "soft64.cuh"

namespace b3g {

constexpr uint32_t kTipBit = 0x80000000u;
constexpr int kMaxStates = 20;
constexpr int kMaxCategories = 16;
constexpr uint32_t kPatternAlign = 128;

// Marks of an entry of a depth-first 20-state FP32 list (NodeOp::pad): the
// right child is multiplied first; the second child is the previous entry's
// output.
constexpr uint32_t kS20Swap = 1u, kS20Prev = 2u;

// Shared-memory slot code meaning "global memory only" (run walk).
constexpr uint32_t kNoSlot = 0xFFu;

// Schedule of the four-state FP32 depth-first walk (tree4.cuh).
constexpr uint32_t kTreeInA = 1u, kTreeInB = 2u; // the child is no tip
constexpr uint32_t kTreePrev = 4u;   // the first child is the previous output
constexpr uint32_t kTreeMemA = 8u, kTreeMemB = 16u; // read from global memory
constexpr uint32_t kTreeKeep = 32u;    // the output goes to its slot
constexpr uint32_t kTreeBarrier = 64u; // a phase ends behind the entry
constexpr uint32_t kTreeCleanA = 1u, kTreeCleanB = 2u; // (more) copied to its slot
// the kinds with code of their own
constexpr uint32_t kTreeKind = kTreeInA | kTreeInB | kTreePrev | kTreeMemA | kTreeMemB;
constexpr uint32_t kTreeTipTip = 0u, kTreePrevTip = kTreeInA | kTreePrev;
// Leaves are given as tile times their number where the tip codes are in
// shared memory, a slot or memory child as the row behind them (else kTreeNoTip).
constexpr uint32_t kTreeNoTip = 0xFFFFFFFFu;
struct __align__(16) TreeOp {
	uint32_t out;
	uint32_t code;     // flags above, the output's slot (bits 8-15), and the base
			   // of the next entry's second child (16-31): 16-byte units
			   // in its category's part of shared memory
	uint32_t next_a;   // the next entry's first child's leaf
	uint32_t after_b;  // the second child's leaf of the entry after that
	uint32_t id[2];    // the children's partials slots
	uint32_t more;     // clean children, the children's slots (8-15, 16-23)
	uint32_t barriers; // phases that end behind the entry
};
// What entry 0 finds in the words before it in the others' case.
struct TreeHead {
	uint32_t tip[3];   // first child's leaf, second's, entry 1's second's
	uint32_t base;
	uint32_t barriers; // phases without an entry before it
};
constexpr uint32_t kTreeChunk = 4;   // entries copied together
constexpr uint32_t kTreeRing = 4 * kTreeChunk; // entries in a group's ring

// One entry of the children-first schedule: output slot and the two
// children, each either a partial slot or (kTipBit | leaf id).
struct NodeOp {
	uint32_t out;
	uint32_t left;
	uint32_t right;
	uint32_t pad;
};

// Substitution model resident on the device, written by the host (the
// eigensystem is given or decomposed on the host); matrices row-major with
// row stride `states`.
struct ModelDev {
	double V[kMaxStates * kMaxStates];
	double Vinv[kMaxStates * kMaxStates];
	double lambda[kMaxStates];
	double Q[kMaxStates * kMaxStates];
	double pi[kMaxStates];
	double cat_rates[kMaxCategories];
	uint32_t shortcuts;
	uint32_t states;
};

struct PtabParams {
	const double *lengths;  // [n][2] time lengths, or null
	const double *matrices; // [n][2][C][S][S], or null
	const ModelDev *model;
	double clock_rate;
	uint32_t n;
	uint32_t C;
	void *ptab; // R [n][2][C][S+1][S]
	SoftTab4 *soft; // [n][2][C] beside the four-state FP64 tables, or null
	void *soft20;   // [n][2][C] beside the 20-state ones (SoftTab20)
};

constexpr uint32_t kScalePow = 8;

struct PruneParams {
	const uint8_t *tips;
	void *partials;
	int32_t *scales;
	const NodeOp *ops;
	const void *ptab;
	const SoftTab4 *soft; // four-state FP64 form: the tables as integers, or
			      // null (the caller's own tables: plain walk)
	// depth-first order (four-state FP64 and 20-state FP32 walks): with
	// `groups` > 1 the list has `phases`; in phase ph group g of a block
	// walks entries [segs[ph groups + g], segs[ph groups + g + 1])
	const uint32_t *segs;
	uint32_t groups, phases;
	// 20-state FP64 form: its integer tables, and the root's value and
	// count [C][ldp] (ticket then holds a counter a 64-pattern tile)
	const void *soft20;
	double *root_val;
	int32_t *root_exp;
	const double *pi;
	const uint32_t *weights;
	double *site_lnl;   // [ldp]
	double *cat_lnl;    // [C][ldp] or null
	double *block_sums; // [gridDim.x]
	unsigned *ticket;   // zero between launches
	double *lnl_out;    // [1]
	double *lnl_host;   // host-mapped word that also receives it, or null
	// host-mapped [gridDim.x], or null: each block writes its sum there and
	// the host folds them (no ticket, no last-block fold, no lnl_out)
	double *sums_host;
	uint32_t n;
	uint32_t ldp;
	uint32_t C;
	uint32_t scale_ln;
	uint32_t num_leaves; // rows of tips
	uint32_t tips_smem;  // stage the block's tip codes in shared memory
	// 64-bit element indices whatever num_leaves says (the slot ids come
	// from a caller whose buffers may hold more than 2 * num_leaves slots)
	uint32_t wide_index;
	// run-synchronous walk (prune4_runs_kernel): runs[0..n_runs] are the
	// first entries of the runs of mutually independent entries, then n
	const uint32_t *runs;
	uint32_t n_runs;
	uint32_t tile; // patterns per tile
	uint32_t ptab_smem; // stage the transition tables in shared memory
	// per entry: shared-memory slot of the output (bits 0-7) and of the
	// left (8-15) and right (16-23) child, kNoSlot where the value lives
	// in global memory only; null or n_slots 0: no slots
	const uint32_t *slots;
	uint32_t n_slots;
	// run walk that builds its own transition tables (tables_inline):
	// run r + 1's tables are built while run r is walked, into a double
	// buffer of max_run entries in shared memory, with ptab4_kernel's
	// arithmetic, from the edge lengths (or the given matrices)
	const ModelDev *model;
	const double *lengths;  // [n][2], or null
	const double *matrices; // [n][2][C][4][4], or null
	double clock_rate;
	uint32_t tables_inline;
	uint32_t max_run;
	uint32_t lengths_smem; // stage the lengths in shared memory
	double scale_threshold;
	double scale_mult;
	// e^(-scale_ln d) for d = 1 ..., or zeros: the FP64 form's root mixes the
	// categories with them
	double scale_pow[kScalePow];
	double log_inv_c;
};

// One member of a batch (many calculators evaluated by one launch).  The
// pointers are the member's own device store; written once per batch.
struct MemberDesc {
	const uint8_t *tips;
	float *partials;     // FP32 chosen form
	int32_t *scales;
	float *ptab;
	const uint8_t *stage; // the member's staged block (ops, pi, runs, lengths)
	const ModelDev *model;
	const uint32_t *weights;
	double *site_lnl;
	double *tile_sums;   // one per tile, owned by the batch
	unsigned *ticket;    // tiles finished, owned by the batch
	uint32_t off_pi, off_runs, off_in, off_tree;
	uint32_t ldp, C, L, tile;
	double log_inv_c;
};

// The run walk; the short-list kernel (n <= kDirectMax, C of 1, 2 or 4); the
// depth-first walk (other single-tree lists).
constexpr uint32_t kListRuns = 0, kListShort = 1, kListTree = 2;
// Shared memory of a block of the batched depth-first walk: beside it fits one
// block of the short-list kernel.
constexpr uint32_t kBatchTreeSmem = 144u * 1024u;

// Per step and member, written by the host before every batched launch.
struct MemberStep {
	uint32_t n;      // dirty entries (0: nothing to evaluate)
	uint32_t n_runs;
	uint32_t tips_smem;
	uint32_t tile; // patterns per tile for this step (divides ldp)
	uint32_t fold; // the member's own tile, a multiple of it: order of the sum
	uint32_t kind; // the kernel that walks the list
	// a depth-first list's schedule (kListTree)
	uint32_t groups, phases, n_slots, clean;
	double clock_rate;
};

struct BatchParams {
	const MemberDesc *members;
	const MemberStep *steps;
	double *lnl_out;     // [members]
	unsigned *work_next; // work counters, zero before each launch: [0] the
			     // run walk's, [1..3] the short-list kernels' (4,
			     // 2 and 1 categories)
	uint32_t num_members;
	uint32_t smem_ops_bytes;  // shared memory reserved for ops + runs
	uint32_t smem_tips_bytes; // shared memory reserved for a tip tile
	uint32_t max_cols;
	uint32_t narrow; // every member indexes with 32 bits
	uint32_t smem_ptab_bytes; // shared memory reserved for staged tables
};

// A run of the schedule holds at most kRunCap / C entries (at least 8):
// the run walk builds one run's transition tables in shared memory.
constexpr uint32_t kRunCap = 128;

// Transition tables of one list fit shared memory at most this large.
constexpr uint32_t kPtabSmemBytes = 32u * 1024u;

// Fused single-launch evaluation of a short list (FP32 chosen form, four
// states, one, two or four categories): the schedule, the edge lengths and the root
// frequencies travel in the kernel parameters, so the launch needs no
// upload, no transition kernel and no read-back copy.
constexpr uint32_t kDirectMax = 48; // entries
struct DirectParams {
	const uint8_t *tips;
	void *partials;
	int32_t *scales;
	const uint32_t *weights;
	const ModelDev *model;
	double *site_lnl;   // [ldp]
	double *block_sums; // [gridDim.x]
	unsigned *ticket;   // zero between launches
	double *lnl_out;    // device copy of the result
	double *lnl_host;   // host-mapped pinned word, written by the last block
			    // (without a host fold)
	// host-mapped [gridDim.x], or null: each block writes its sum there and
	// the host folds them (then lnl_out and lnl_host are not written)
	double *sums_host;
	uint32_t n, ldp, L, C; // C: 1, 2 or 4 categories
	double clock_rate;
	double log_inv_c;
	double pi[4];
	// the model as the table builder reads it, converted on the host with
	// the same rounding: V, V^-1, lambda in FP32, the shortcuts flag at
	// [36]; and clock rate x category rate in FP64 (the model in global
	// memory is read only on the shortcut paths)
	float eig[40];
	double rate[4];
	// pad: where the left (bits 0-7) and right (8-15) child comes from (kSrc*)
	NodeOp ops[kDirectMax];
	double lengths[2 * kDirectMax]; // [n][2] time lengths
};

// Sources of a child in the fused short-list walk, set by the host: a tip
// code, a clean partial (not an output of this list: loaded ahead), the
// previous or the second previous entry's output (registers), or an older
// output of this list (read back when needed).
enum : uint8_t { kSrcTip = 0, kSrcClean, kSrcPrev, kSrcPrev2, kSrcEarlier };

// Launchers (kernels4.cu).  Each returns the launch error.
cudaError_t launch_ptab4(const PtabParams &p, bool f32, cudaStream_t s);
cudaError_t launch_prune4(const PruneParams &p, bool f32, uint32_t tile,
			  cudaStream_t s);
// Run-synchronous FP32 walk: `ctas` persistent blocks over ldp / p.tile
// pattern tiles.  Needs p.runs; block sums sized for `ctas`.
// The depth-first FP32 walk (tree4.cuh): `tile` patterns (64 or 128) a block,
// `groups` x C warps (at most 16); needs ptab, sums_host, and the schedule for n_slots
// shared-memory slots, group after group.  segs: the groups' first entries, n,
// then their heads.
size_t prune4_tree_smem(const PruneParams &p);
// bases (16-byte units in a category's part of shared memory) of the second
// child's rows of a group's entry k, and of a slot's vectors
uint32_t prune4_tree_entry(uint32_t group, uint32_t k);
uint32_t prune4_tree_slot(uint32_t groups, uint32_t tile, uint32_t slot);
cudaError_t launch_prune4_tree(const PruneParams &p, bool clean, cudaStream_t s);
cudaError_t launch_ptab4_rows(const PtabParams &p, cudaStream_t s);

// dynamic shared memory of prune4_runs_kernel for these parameters
size_t prune4_runs_smem(const PruneParams &p);
// block: 512 (two blocks per SM) or 1024 threads (one per SM)
cudaError_t launch_prune4_runs(const PruneParams &p, uint32_t ctas,
			       uint32_t block, cudaStream_t s);
// 20-state tensor-core path (prune20tc.cuh), FP32 chosen form.
struct Tc20Params {
	const uint8_t *tips;
	float *partials;
	int32_t *scales;
	const NodeOp *ops;
	const float *tab;    // [n][2][C][21][20] tip rows
	const float *tc_tab; // [n][2][C][2][768] hi/lo MMA operand blocks
	const double *pi;
	const uint32_t *weights;
	double *root_val;    // [C][ldp] pi . x at the root
	int32_t *root_exp;   // [C][ldp] its power-of-two exponent
	double *site_lnl;    // [ldp]
	double *cat_lnl;     // [C][ldp] or null
	double *block_sums;  // [ldp / 128]
	unsigned *ticket;    // zero between launches
	double *lnl_out;
	unsigned *status;    // set to 1 when a bounded tensor-core wait gave up
	uint32_t n, ldp, C, L;
	uint32_t ops_smem;   // stage the list in shared memory
	uint32_t tips_smem;  // stage the tile's tip codes in shared memory
	uint32_t groups;     // 128-thread groups per CTA (1 or 2)
	uint32_t cluster;    // CTAs per (tile, category) work item, 1..8
	double log_inv_c;
};
// Dynamic shared memory of one tensor-core pruning CTA.
size_t prune20tc_smem(uint32_t groups, bool ops_smem, uint32_t n, bool tips_smem,
		      uint32_t L);
// Tables of both kinds for the tensor-core path: p.ptab receives the FP32
// tip rows, tc_tab the operand blocks.
cudaError_t launch_ptab20tc(const PtabParams &p, float *tc_tab, cudaStream_t s);
// Pruning (one CTA of p.groups x 128 threads per 128-pattern tile and
// category, 4 / p.groups CTAs per SM) then the root's category mixing and
// fold.
cudaError_t launch_prune20tc(const Tc20Params &p, cudaStream_t s);
// 20-state path: transition tables [n][2][C][21][20] computed in FP64 (FP64
// form: and their integer form, soft_tab20_bytes() each).
cudaError_t launch_ptab20(const PtabParams &p, bool f32, cudaStream_t s);
size_t soft_tab20_bytes();
// FP32 form with register MMAs (prune20.cuh): a block of p.groups (1..4)
// warps per 32-pattern tile and category; needs root buffers, sums_host (a
// sum a tile), zeroed tickets (one a tile), marked entries and, with several
// groups, segs.
cudaError_t launch_prune20(const PruneParams &p, cudaStream_t s);
// Words of prm.segs that a block's shared memory holds beside the rest (kSegSmem
// in all, the default limit less room for a few static words): the four-state
// FP64 walk with `warps` warps a block, the 20-state FP32 walk with `groups`.
constexpr uint32_t kSegSmem = 48u * 1024u - 64u;
uint32_t prune4_f64_seg_words(uint32_t warps);
uint32_t prune20_seg_words(uint32_t groups);
// Blocks of `groups` warps of that walk that one SM holds.
uint32_t prune20_blocks_per_sm(uint32_t groups);
// FP64 form (prune20f64.cuh): a block of `groups` (1..4) x 128 threads per
// 64-pattern tile and category; needs soft20, runs, root buffers, sums_host
// (a sum a tile) and zeroed tickets (one a tile).
cudaError_t launch_prune20_f64(const PruneParams &p, uint32_t groups, cudaStream_t s);
// Fused short-list evaluation: `ctas` persistent blocks over ldp / 128
// pattern tiles; needs p.n <= kDirectMax and block sums sized for `ctas`.
cudaError_t launch_prune4_direct(const DirectParams &p, uint32_t ctas,
				 cudaStream_t s);
// Batched evaluation (FP32): transition tables of every member with work,
// then one persistent pruning launch over all members' pattern tiles.
// max_entries = largest member n * 2 * C.
cudaError_t launch_ptab4_batch(const BatchParams &p, uint32_t max_entries,
			       cudaStream_t s);
cudaError_t launch_prune4_tree_batch(const BatchParams &p, uint32_t ctas, cudaStream_t s);
cudaError_t launch_prune4_batch(const BatchParams &p, uint32_t ctas,
				cudaStream_t s);
// Batched short lists: every member whose step is direct and has C
// categories (1, 2 or 4), `ctas` persistent blocks taking (member, tile)
// items from that category count's counter.
cudaError_t launch_prune4_direct_batch(const BatchParams &p, uint32_t C,
				       uint32_t ctas, cudaStream_t s);

} // namespace b3g
