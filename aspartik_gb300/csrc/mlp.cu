// mlp.cu -- training and inference kernels of the delayed-acceptance
// surrogate (see mlp.hpp).
//
// Layers are stored flat, layer l as W_l [out][in] row-major followed by
// b_l [out].  Hidden layers use GELU in its tanh form (Hendrycks and
// Gimpel, "Gaussian Error Linear Units", 2016):
//     gelu(x) = x/2 (1 + tanh(u)),  u = sqrt(2/pi) (x + 0.044715 x^3).
// A training step is seven launches: three hidden layers forward, the pair
// objective with the output layer's backward pass, and three hidden layers
// backward; Adam (Kingma and Ba, 2015) updates the parameters.
#include <cooperative_groups.h>

#include "calculator.hpp"
#include "mlp.hpp"

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>
#include <numeric>
#include <random>
#include <type_traits>

namespace b3g {
namespace {

namespace cg = cooperative_groups;

constexpr float kGeluC = 0.7978845608028654f; // sqrt(2 / pi)
constexpr float kGeluA = 0.044715f;

__device__ __forceinline__ float gelu(float x)
{
	const float u = kGeluC * (x + kGeluA * x * x * x);
	return 0.5f * x * (1.0f + tanhf(u));
}

__device__ __forceinline__ float gelu_grad(float x)
{
	const float u = kGeluC * (x + kGeluA * x * x * x);
	const float t = tanhf(u);
	return 0.5f * (1.0f + t) +
	       0.5f * x * (1.0f - t * t) * kGeluC * (1.0f + 3.0f * kGeluA * x * x);
}

// ---------------------------------------------------------------------------
// FP32 matrix products of the training step.
//
// A block of 256 threads computes a 32 x 64 tile of C[m][n] = sum_k A'(m, k)
// B'(k, n): two halves of 128 threads, a thread 4 x 4 products over its
// half's 16 of every 32 k, the halves added at the end (each keeps two of
// the four rows), or (kHalves false) 2 x 4 products over every k in order;
// operand tiles of 32 k pass through three shared-memory buffers filled by
// cp.async two ahead of their use.  A'(m, k) = TA ? A[k][m] : A[m][k] with row
// stride lda, B'(k, n) = TB ? B[n][k] : B[k][n] with row stride ldb.  The tile
// is this small because the step is: 1,024 rows x 256 units are 128 tiles for
// 152 SMs, and 256 threads because one warp a scheduler waits on its own
// loads (16 x 16 tiles with one product a thread and shared-memory word pair
// took 17 to 36 us a product, 128 threads 9.7, two halves 6, 256 threads over
// every k 7).
constexpr uint32_t kTm = 32, kTn = 64, kTk = 32, kTt = 256; // kTt: threads
constexpr uint32_t kTs = 3; // buffers
// a weight gradient's rows are split over up to kSplits blocks a tile, at
// least kSplitRows each, whose partial tiles the last one adds in a fixed order
constexpr uint32_t kSplits = 16, kSplitRows = 128;

struct MlpSmem {
	// [m][k] or [k][m], rows padded to 36 / 68 floats (16-byte aligned)
	float a[kTs][kTk * (kTm + 4)];
	float b[kTs][kTn * (kTk + 4)];
};

__device__ __forceinline__ void mlp_cp16(float *dst, const float *src, bool live)
{
	asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(
			     (uint32_t)__cvta_generic_to_shared(dst)),
		     "l"(src), "r"(live ? 16 : 0)
		     : "memory");
}
__device__ __forceinline__ void mlp_cp4(float *dst, const float *src, bool live)
{
	asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(
			     (uint32_t)__cvta_generic_to_shared(dst)),
		     "l"(src), "r"(live ? 4 : 0)
		     : "memory");
}

// rows x cols of a row-major matrix from (r0, c0), elements outside [0, R) x
// [0, C) as zero, into dst with row stride `pitch`.  vec: ld, c0, C and the
// base are multiples of four floats.
template <uint32_t rows, uint32_t cols>
__device__ __forceinline__ void mlp_tile(float *dst, uint32_t pitch, const float *src,
					 uint32_t r0, uint32_t c0, uint32_t R, uint32_t C,
					 uint32_t ld, bool vec)
{
	if (vec) {
#pragma unroll
		for (uint32_t i = 0; i < rows * cols / 4 / kTt; ++i) {
			const uint32_t at = threadIdx.x + kTt * i;
			const uint32_t r = at / (cols / 4), c = 4 * (at % (cols / 4));
			const bool live = r0 + r < R && c0 + c < C;
			mlp_cp16(dst + r * pitch + c,
				 live ? src + (size_t)(r0 + r) * ld + c0 + c : src, live);
		}
	} else {
#pragma unroll 4
		for (uint32_t i = 0; i < rows * cols / kTt; ++i) {
			const uint32_t at = threadIdx.x + kTt * i;
			const uint32_t r = at / cols, c = at % cols;
			const bool live = r0 + r < R && c0 + c < C;
			mlp_cp4(dst + r * pitch + c,
				live ? src + (size_t)(r0 + r) * ld + c0 + c : src, live);
		}
	}
}

__device__ __forceinline__ bool mlp_vec(const float *p, uint32_t ld)
{
	return (ld & 3u) == 0 && ((uintptr_t)p & 15u) == 0;
}

// The tile's products over k in [k0, k1).  Thread (h, ty, tx) leaves with rows
// 4 ty + 2 h + i, columns TB ? tx + 16 j : 4 tx + j in acc[i][j].  col_sum (TA): threads 0..31 also add
// A'(m0 + thread, k) over k.
template <bool TA, bool TB, bool kHalves = true>
__device__ __forceinline__ void mlp_product(MlpSmem &sm, const float *A, const float *B,
					    uint32_t m0, uint32_t n0, uint32_t M, uint32_t N,
					    uint32_t k0, uint32_t k1, uint32_t lda, uint32_t ldb,
					    float acc[2][4], float *col_sum = nullptr)
{
	constexpr uint32_t pa = TA ? kTm + 4 : kTk + 4, pb = TB ? kTk + 4 : kTn + 4;
	const uint32_t tx = threadIdx.x & 15u, ty = (threadIdx.x >> 4) & 7u, h = threadIdx.x >> 7;
	constexpr int kRows = kHalves ? 4 : 2; // a thread's rows, from row 4 ty (+ 2 h)
	const uint32_t r0 = 4 * ty + (kHalves ? 0u : 2 * h);
	float c[kRows][4];
	// a row of the operand in memory must be whole vectors up to its end
	const bool va = mlp_vec(A, lda) && ((TA ? M : k1) & 3u) == 0;
	const bool vb = mlp_vec(B, ldb) && ((TB ? k1 : N) & 3u) == 0;
	auto fetch = [&](uint32_t k, uint32_t buf) {
		if (k < k1) {
			if (TA)
				mlp_tile<kTk, kTm>(sm.a[buf], pa, A, k, m0, k1, M, lda, va);
			else
				mlp_tile<kTm, kTk>(sm.a[buf], pa, A, m0, k, M, k1, lda, va);
			if (TB)
				mlp_tile<kTn, kTk>(sm.b[buf], pb, B, n0, k, N, k1, ldb, vb);
			else
				mlp_tile<kTk, kTn>(sm.b[buf], pb, B, k, n0, k1, N, ldb, vb);
		}
		asm volatile("cp.async.commit_group;" ::: "memory");
	};
#pragma unroll
	for (int i = 0; i < kRows; ++i)
#pragma unroll
		for (int j = 0; j < 4; ++j)
			c[i][j] = 0.0f;
	float cs = 0.0f;
	for (uint32_t q = 0; q + 1 < kTs; ++q)
		fetch(k0 + q * kTk, q);
	uint32_t buf = 0, next = kTs - 1;
	for (uint32_t k = k0; k < k1; k += kTk) {
		asm volatile("cp.async.wait_group %0;" ::"n"(kTs - 2) : "memory");
		__syncthreads(); // this tile is there, the one before it used up
		fetch(k + (kTs - 1) * kTk, next);
		const float *sa = sm.a[buf], *sb = sm.b[buf];
#pragma unroll
		for (uint32_t k4 = 0; k4 < (kHalves ? kTk / 2 : kTk); k4 += 4) {
			const uint32_t kk = kHalves ? h * (kTk / 2) + k4 : k4;
			float a[4][4], b[4][4]; // [k][i], [k][j]
#pragma unroll
			for (int i = 0; i < 4; ++i) {
				if (TA) {
					const float4 v = *reinterpret_cast<const float4 *>(
						sa + (kk + i) * pa + 4 * ty);
					a[i][0] = v.x, a[i][1] = v.y, a[i][2] = v.z, a[i][3] = v.w;
				} else if (i < kRows) {
					const float4 v = *reinterpret_cast<const float4 *>(
						sa + (r0 + i) * pa + kk);
					a[0][i] = v.x, a[1][i] = v.y, a[2][i] = v.z, a[3][i] = v.w;
				}
				if (TB) {
					const float4 v = *reinterpret_cast<const float4 *>(
						sb + (tx + 16 * i) * pb + kk);
					b[0][i] = v.x, b[1][i] = v.y, b[2][i] = v.z, b[3][i] = v.w;
				} else {
					const float4 v = *reinterpret_cast<const float4 *>(
						sb + (kk + i) * pb + 4 * tx);
					b[i][0] = v.x, b[i][1] = v.y, b[i][2] = v.z, b[i][3] = v.w;
				}
			}
#pragma unroll
			for (int q = 0; q < 4; ++q)
#pragma unroll
				for (int i = 0; i < kRows; ++i)
#pragma unroll
					for (int j = 0; j < 4; ++j)
						c[i][j] = fmaf(a[q][i], b[q][j], c[i][j]);
		}
		if (TA && col_sum && threadIdx.x < kTm)
			for (uint32_t kk = 0; kk < kTk; ++kk)
				cs += sa[kk * pa + threadIdx.x];
		buf = buf + 1 == kTs ? 0 : buf + 1;
		next = next + 1 == kTs ? 0 : next + 1;
	}
	__syncthreads(); // the buffers are free
	if (TA && col_sum)
		*col_sum = cs;
	if constexpr (!kHalves) {
		static_assert(!TA || kHalves, "whole k: rows of A' only");
#pragma unroll
		for (int i = 0; i < 2; ++i)
#pragma unroll
			for (int j = 0; j < 4; ++j)
				acc[i][j] = c[i][j];
		return;
	} else {
		// the other half's sums of this thread's rows, through shared memory
		float4 *ex = reinterpret_cast<float4 *>(&sm);
#pragma unroll
		for (int i = 0; i < 2; ++i) {
			const int o = 2 * (1 - (int)h) + i; // what the other half keeps
			const float *v = o == 0 ? c[0] : o == 1 ? c[1] : o == 2 ? c[2] : c[3];
			ex[(threadIdx.x ^ 128u) + kTt * i] = make_float4(v[0], v[1], v[2], v[3]);
		}
		__syncthreads();
#pragma unroll
		for (int i = 0; i < 2; ++i) {
			const float4 v = ex[threadIdx.x + kTt * i];
			const float *w = h ? c[2 + i] : c[i];
			acc[i][0] = w[0] + v.x;
			acc[i][1] = w[1] + v.y;
			acc[i][2] = w[2] + v.z;
			acc[i][3] = w[3] + v.w;
		}
	}
}

// Hidden layer: z = x W^T + b and a = gelu(z), each product one chain over k in
// order (not halves): the residuals, whose rounding the output bias's gradient
// consists of (below), do not depend on the tiling.  Grid (N / 64, M / 32).
__global__ void __launch_bounds__(kTt) mlp_forward_kernel(const float *__restrict__ x,
							   const float *__restrict__ W,
							   const float *__restrict__ bias,
							   float *__restrict__ z,
							   float *__restrict__ a, uint32_t M,
							   uint32_t N, uint32_t K)
{
	__shared__ __align__(16) MlpSmem sm;
	const uint32_t m0 = blockIdx.y * kTm, n0 = blockIdx.x * kTn;
	const uint32_t tx = threadIdx.x & 15u;
	const uint32_t row = 4 * ((threadIdx.x >> 4) & 7u) + 2 * (threadIdx.x >> 7);
	float acc[2][4];
	mlp_product<false, true, false>(sm, x, W, m0, n0, M, N, 0, K, K, K, acc);
#pragma unroll
	for (int j = 0; j < 4; ++j) {
		const uint32_t n = n0 + tx + 16 * j;
		if (n >= N)
			continue;
		const float bn = bias[n];
#pragma unroll
		for (int i = 0; i < 2; ++i) {
			const uint32_t m = m0 + row + i;
			if (m >= M)
				continue;
			const float v = acc[i][j] + bn;
			z[(size_t)m * N + n] = v;
			a[(size_t)m * N + n] = gelu(v);
		}
	}
}

// Sum over lanes of a warp, the same in every lane, in a fixed order.
__device__ __forceinline__ float warp_sum(float v)
{
	for (int off = 16; off > 0; off >>= 1)
		v += __shfl_xor_sync(0xffffffffu, v, off);
	return v;
}

// y[m] = a[m] . w + b, a warp a row (forward pass only).
__global__ void __launch_bounds__(256) mlp_out_kernel(const float *__restrict__ a,
						       const float *__restrict__ w,
						       float *__restrict__ y, uint32_t rows,
						       uint32_t H)
{
	const uint32_t lane = threadIdx.x & 31u, m = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
	if (m >= rows)
		return;
	float v = 0.0f;
	for (uint32_t k = lane; k < H; k += 32)
		v = fmaf(a[(size_t)m * H + k], w[k], v);
	v = warp_sum(v);
	if (lane == 0)
		y[m] = v + w[H];
}

// The pair objective and the last layer's backward pass.  Row i of n holds
// x_new's third layer, row n + i x_old's; a warp a pair: r = y_new - y_old -
// delta, the loss's share r^2, dL/dy = +-2 r / n (dys: the new rows'), and dZ
// of the third layer = dL/dy w gelu'(z).  The last block to finish adds the
// loss shares in block order.  y is one chain over the units in order, then
// the bias, as a forward product forms it: the output layer's gradients are
// small differences of large sums, and hold each value's rounding.
constexpr uint32_t kHeadPairs = 4;
// floats of a staged row: up to 256 units, the eight gradients a lane keeps in
// registers; above, two lanes read their rows in place (a training step of 512
// pairs: 256 units 130 us, 288 156; with plain 16 x 16 products 405 and 454)
__host__ __device__ constexpr uint32_t head_row(uint32_t H)
{
	return H <= 256 ? (H + 3u) & ~3u : 0u;
}
__global__ void __launch_bounds__(32 * kHeadPairs) mlp_head_kernel(
	const float *__restrict__ a, const float *__restrict__ z, const float *__restrict__ w,
	const float *__restrict__ delta, float *__restrict__ dz, float *__restrict__ dys,
	float *__restrict__ losses, float *__restrict__ loss, unsigned *ticket, uint32_t n,
	uint32_t H)
{
	extern __shared__ __align__(16) float sh[]; // [w: Hs][kHeadPairs][2][Hs], H <= 256
	__shared__ float s_loss[kHeadPairs];
	__shared__ unsigned s_last;
	const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
	const uint32_t i = blockIdx.x * kHeadPairs + warp, Hs = head_row(H);
	float *rows = sh + (2 * warp + 1) * Hs; // this warp's new and old row
	if (Hs)
		for (uint32_t k = threadIdx.x; k < H; k += blockDim.x)
			sh[k] = w[k];
	__syncthreads();
	auto value = [&](const float *row, const float *ww) {
		float acc = 0.0f;
		uint32_t k = 0;
		if (Hs)
#pragma unroll 8
			for (; k + 4 <= H; k += 4) {
				const float4 x = *reinterpret_cast<const float4 *>(row + k);
				const float4 y = *reinterpret_cast<const float4 *>(ww + k);
				acc = fmaf(x.x, y.x, acc);
				acc = fmaf(x.y, y.y, acc);
				acc = fmaf(x.z, y.z, acc);
				acc = fmaf(x.w, y.w, acc);
			}
#pragma unroll 16
		for (; k < H; ++k)
			acc = fmaf(row[k], ww[k], acc);
		return acc + w[H];
	};
	float r = 0.0f;
	if (i < n) {
		const float *an = a + (size_t)i * H, *ao = a + (size_t)(n + i) * H;
		const float *zn = z + (size_t)i * H, *zo = z + (size_t)(n + i) * H;
		float gn[8], go[8];
		float f = 0.0f;
		if (Hs) {
			// everything that does not need dL/dy first
#pragma unroll
			for (int q = 0; q < 8; ++q) {
				const uint32_t k = lane + 32 * q;
				const bool live = k < H;
				gn[q] = live ? zn[k] : 0.0f;
				go[q] = live ? zo[k] : 0.0f;
				if (live) {
					rows[k] = an[k];
					rows[Hs + k] = ao[k];
				}
			}
			__syncwarp();
			if (lane < 2)
				f = value(rows + lane * Hs, sh);
#pragma unroll
			for (int q = 0; q < 8; ++q) {
				gn[q] = gelu_grad(gn[q]);
				go[q] = gelu_grad(go[q]);
			}
		} else if (lane < 2) {
			f = value(lane ? ao : an, w);
		}
		r = __shfl_sync(0xffffffffu, f, 0) - __shfl_sync(0xffffffffu, f, 1) - delta[i];
		const float dy = 2.0f * r / n;
		if (lane == 0)
			dys[i] = dy;
		if (Hs) {
#pragma unroll
			for (int q = 0; q < 8; ++q) {
				const uint32_t k = lane + 32 * q;
				if (k < H) {
					dz[(size_t)i * H + k] = dy * sh[k] * gn[q];
					dz[(size_t)(n + i) * H + k] = -dy * sh[k] * go[q];
				}
			}
		} else {
			for (uint32_t k = lane; k < H; k += 32) {
				dz[(size_t)i * H + k] = dy * w[k] * gelu_grad(zn[k]);
				dz[(size_t)(n + i) * H + k] = -dy * w[k] * gelu_grad(zo[k]);
			}
		}
	}
	if (lane == 0)
		s_loss[warp] = r * r;
	__syncthreads();
	if (threadIdx.x == 0) {
		float v = 0.0f;
		for (uint32_t q = 0; q < kHeadPairs; ++q)
			v += s_loss[q];
		losses[blockIdx.x] = v;
		__threadfence();
		s_last = atomicAdd(ticket, 1u) == gridDim.x - 1u;
	}
	__syncthreads();
	if (!s_last || warp != 0)
		return;
	__threadfence();
	float v = 0.0f;
	for (uint32_t k = lane; k < gridDim.x; k += 32)
		v += __ldcg(losses + k);
	v = warp_sum(v);
	if (lane == 0) {
		*loss = v / n;
		*ticket = 0u;
	}
}

// Sums over the rows, one chain in row order, of columns c0 .. c0 + 15 of src
// [R][C]: with dys the rows weighted by +dys[row] (first half) and -dys[row -
// R / 2], and their own sum in *weights.  128 rows a tile, three tiles ahead
// (tiles of 64 columns and 32 rows, two ahead, took 35 us for 1,024 rows: a
// memory latency a tile).
constexpr uint32_t kChainCols = 16, kChainRows = 128, kChainTiles = 4;
__device__ __forceinline__ void mlp_column_chain(MlpSmem &sm, const float *src, uint32_t c0,
						 uint32_t R, uint32_t C, const float *dys,
						 float *out, float *weights)
{
	constexpr uint32_t kTile = kChainRows * kChainCols;
	static_assert(kChainTiles * (kTile + kChainRows) * sizeof(float) <= sizeof(MlpSmem), "");
	float *tiles = reinterpret_cast<float *>(&sm), *scales = tiles + kChainTiles * kTile;
	const uint32_t t = threadIdx.x, n = R / 2;
	const bool vec = mlp_vec(src, C);
	auto fetch = [&](uint32_t k, uint32_t buf) {
		if (k < R) {
			mlp_tile<kChainRows, kChainCols>(tiles + buf * kTile, kChainCols, src, k, c0,
							 R, C, C, vec);
			const uint32_t row = k + t;
			if (dys && t < kChainRows)
				mlp_cp4(scales + buf * kChainRows + t,
					dys + (row < n ? row : row < R ? row - n : 0u), row < R);
		}
		asm volatile("cp.async.commit_group;" ::: "memory");
	};
	for (uint32_t q = 0; q + 1 < kChainTiles; ++q)
		fetch(q * kChainRows, q);
	float acc = 0.0f;
	uint32_t buf = 0;
	for (uint32_t k = 0; k < R; k += kChainRows) {
		asm volatile("cp.async.wait_group %0;" ::"n"(kChainTiles - 2) : "memory");
		__syncthreads(); // this tile is there, the one before it used up
		fetch(k + (kChainTiles - 1) * kChainRows, (buf + kChainTiles - 1) % kChainTiles);
		const float *v = tiles + buf * kTile + t, *w = scales + buf * kChainRows;
		const uint32_t rows = min(kChainRows, R - k);
		if (t < kChainCols) {
			if (!dys) {
#pragma unroll 16
				for (uint32_t r = 0; r < rows; ++r)
					acc += v[r * kChainCols];
			} else {
#pragma unroll 16
				for (uint32_t r = 0; r < rows; ++r)
					acc = fmaf(k + r < n ? w[r] : -w[r], v[r * kChainCols], acc);
			}
		} else if (t == 32 && weights) {
#pragma unroll 16
			for (uint32_t r = 0; r < rows; ++r)
				acc += k + r < n ? w[r] : -w[r];
		}
		buf = (buf + 1) % kChainTiles;
	}
	if (t < kChainCols && c0 + t < C)
		out[c0 + t] = acc;
	else if (t == 32 && weights)
		*weights = acc;
}

// One hidden layer's backward pass.  Where dys is given (the last hidden
// layer), first the output layer's gradients and this layer's bias gradient as
// chains over the rows.  Then dw_blocks: the weight gradient dW[o][i] = sum_rows dZ[row][o] a[row][i] and the bias gradient,
// tiles x splits of split_rows rows; with several splits the partial tiles go
// to `part` and a tile's last block adds them in split order.  Then
// da_blocks: dZ of the layer below, (dZ W) gelu'(z_below).
struct MlpBackward {
	const float *dz, *a, *W, *z_below;
	float *dW, *db, *dz_below;
	float *part;       // [tiles][splits][kTm * kTn + kTm]
	unsigned *tickets; // [tiles], zero between launches
	const float *dys, *a_out; // dL/dy, this layer's outputs
	float *head_grad;
	uint32_t rows, O, I, splits, split_rows, dw_blocks, da_blocks;
};
__global__ void __launch_bounds__(kTt) mlp_backward_kernel(MlpBackward p)
{
	__shared__ __align__(16) MlpSmem sm;
	__shared__ unsigned s_last;
	const uint32_t tx = threadIdx.x & 15u;
	const uint32_t row = 4 * ((threadIdx.x >> 4) & 7u) + 2 * (threadIdx.x >> 7);
	float acc[2][4];
	// (the chains first: they are the longest blocks)
	const uint32_t chains = p.dys ? 2 * ((p.O + kChainCols - 1) / kChainCols) : 0u;
	if (blockIdx.x < chains) {
		const uint32_t t = blockIdx.x >> 1;
		if (blockIdx.x & 1u)
			mlp_column_chain(sm, p.dz, t * kChainCols, p.rows, p.O, nullptr, p.db, nullptr);
		else
			mlp_column_chain(sm, p.a_out, t * kChainCols, p.rows, p.O, p.dys, p.head_grad,
					 t == 0 ? p.head_grad + p.O : nullptr);
		return;
	}
	const uint32_t block = blockIdx.x - chains;
	if (block >= p.dw_blocks) {
		const uint32_t t = block - p.dw_blocks, nt = (p.I + kTn - 1) / kTn;
		const uint32_t m0 = t / nt * kTm, n0 = t % nt * kTn;
		mlp_product<false, false>(sm, p.dz, p.W, m0, n0, p.rows, p.I, 0, p.O, p.O, p.I,
					  acc);
#pragma unroll
		for (int i = 0; i < 2; ++i) {
			const uint32_t m = m0 + row + i;
			if (m >= p.rows)
				continue;
#pragma unroll
			for (int j = 0; j < 4; ++j) {
				const uint32_t n = n0 + 4 * tx + j;
				if (n < p.I) {
					const size_t at = (size_t)m * p.I + n;
					p.dz_below[at] = acc[i][j] * gelu_grad(p.z_below[at]);
				}
			}
		}
		return;
	}
	const uint32_t tile = block / p.splits, split = block - tile * p.splits;
	const uint32_t nt = (p.I + kTn - 1) / kTn;
	const uint32_t m0 = tile / nt * kTm, n0 = tile % nt * kTn;
	const uint32_t k0 = split * p.split_rows, k1 = min(p.rows, k0 + p.split_rows);
	const bool bias = n0 == 0 && !p.dys;
	float cs = 0.0f;
	mlp_product<true, false>(sm, p.dz, p.a, m0, n0, p.O, p.I, k0, k1, p.O, p.I, acc,
				 bias ? &cs : nullptr);
	if (p.splits > 1) {
		float *part = p.part + (size_t)tile * p.splits * (kTm * kTn + kTm);
		float4 *mine = reinterpret_cast<float4 *>(part + split * (kTm * kTn + kTm));
#pragma unroll
		for (int i = 0; i < 2; ++i)
			mine[(row + i) * (kTn / 4) + tx] =
				make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
		if (threadIdx.x < kTm)
			reinterpret_cast<float *>(mine)[kTm * kTn + threadIdx.x] = cs;
		__threadfence();
		__syncthreads();
		if (threadIdx.x == 0)
			s_last = atomicAdd(p.tickets + tile, 1u) == p.splits - 1u;
		__syncthreads();
		if (!s_last)
			return;
		__threadfence();
		if (threadIdx.x == 0)
			p.tickets[tile] = 0u;
		cs = 0.0f;
#pragma unroll
		for (int i = 0; i < 2; ++i)
#pragma unroll
			for (int j = 0; j < 4; ++j)
				acc[i][j] = 0.0f;
#pragma unroll 4
		for (uint32_t q = 0; q < p.splits; ++q) {
			const float *from = part + (size_t)q * (kTm * kTn + kTm);
#pragma unroll
			for (int i = 0; i < 2; ++i) {
				const float4 v = __ldcg(reinterpret_cast<const float4 *>(from) +
							(row + i) * (kTn / 4) + tx);
				acc[i][0] += v.x;
				acc[i][1] += v.y;
				acc[i][2] += v.z;
				acc[i][3] += v.w;
			}
			if (threadIdx.x < kTm)
				cs += __ldcg(from + kTm * kTn + threadIdx.x);
		}
	}
#pragma unroll
	for (int i = 0; i < 2; ++i) {
		const uint32_t m = m0 + row + i;
		if (m >= p.O)
			continue;
#pragma unroll
		for (int j = 0; j < 4; ++j) {
			const uint32_t n = n0 + 4 * tx + j;
			if (n < p.I)
				p.dW[(size_t)m * p.I + n] = acc[i][j];
		}
	}
	if (bias && threadIdx.x < kTm && m0 + threadIdx.x < p.O)
		p.db[m0 + threadIdx.x] = cs;
}

__global__ void adam_kernel(float *__restrict__ p, const float *__restrict__ g,
			    float *__restrict__ m, float *__restrict__ v,
			    uint32_t count, float lr, float b1, float b2,
			    float c1, float c2, float eps)
{
	const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
	if (i >= count)
		return;
	const float gi = g[i];
	const float mi = b1 * m[i] + (1.0f - b1) * gi;
	const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
	m[i] = mi;
	v[i] = vi;
	p[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
}

// rows of the dataset gathered by index: out[r] = src[idx[r]]
__global__ void gather_rows_kernel(const float *__restrict__ src,
				   const uint32_t *__restrict__ idx,
				   float *__restrict__ out, uint32_t rows,
				   uint32_t cols)
{
	const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
	if (i >= rows * cols)
		return;
	const uint32_t r = i / cols, c = i - r * cols;
	out[i] = src[(size_t)idx[r] * cols + c];
}

// f(x_new) - f(x_old) for one pair, by a cluster of kDeltaCluster CTAs.
// Every CTA holds all activations of the current layer in shared memory and
// computes its own slice of the next layer's units: warp w of the CTA takes
// kDeltaRows consecutive units at a time and reads their rows of W with all
// loads issued before any product (float4 loads where the rows allow),
// reduces both inputs' dot products across the warp in a fixed order, and
// lanes 0..7 / 8..15 write the two GELU outputs into the eight CTAs' shared
// memory (DSMEM); a cluster barrier ends the layer.  So one inference reads
// its weights through eight SMs instead of one, with many loads in flight
// (one block walking the rows one after another waits an L2 round trip per
// row).  The pair is read from and the result written to host-mapped
// memory: pair = [x_new (in), x_old (in)], result at out (by CTA 0).
constexpr uint32_t kDeltaCluster = 8;
constexpr uint32_t kDeltaRows = 4;

__device__ __forceinline__ float dot4(float4 w, float4 x)
{
	return fmaf(w.x, x.x, fmaf(w.y, x.y, fmaf(w.z, x.z, w.w * x.w)));
}

// One cluster per pair: pair k = pairs[k * stride ...], result out[k].
__global__ void __cluster_dims__(kDeltaCluster, 1, 1) __launch_bounds__(256)
	mlp_delta_kernel(const float *__restrict__ params, const float *pairs, float *out,
			 uint32_t in, uint32_t hidden, uint32_t stride)
{
	extern __shared__ __align__(16) float sh[];
	cg::cluster_group cluster = cg::this_cluster();
	const uint32_t rank = cluster.block_rank();
	const uint32_t item = blockIdx.x / kDeltaCluster;
	const float *pair = pairs + (size_t)item * stride;
	out += item;
	const uint32_t width_max = max(in, hidden);
	float *a = sh;                 // [2][width] current layer (inputs first)
	float *b = sh + 2 * width_max; // [2][hidden] next layer
	const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
	const uint32_t warps = blockDim.x >> 5;
	for (uint32_t k = threadIdx.x; k < 2 * in; k += blockDim.x)
		a[k] = pair[k];
	// this CTA's units of every hidden layer
	const uint32_t per = (hidden + kDeltaCluster - 1) / kDeltaCluster;
	const uint32_t o_begin = rank * per, o_end = min(hidden, o_begin + per);
	cluster.sync(); // every CTA has started before any DSMEM write
	const float *W = params;
	uint32_t width = in;
	for (int layer = 0; layer < 3; ++layer) {
		const float *bias = W + (size_t)hidden * width;
		const bool vec = (width & 3u) == 0 && ((uintptr_t)W & 15u) == 0;
		for (uint32_t o0 = o_begin + warp * kDeltaRows; o0 < o_end;
		     o0 += warps * kDeltaRows) {
			float z0[kDeltaRows], z1[kDeltaRows];
#pragma unroll
			for (uint32_t r = 0; r < kDeltaRows; ++r)
				z0[r] = z1[r] = 0.0f;
			if (vec) {
				for (uint32_t k = 4 * lane; k < width; k += 128) {
					float4 wv[kDeltaRows];
#pragma unroll
					for (uint32_t r = 0; r < kDeltaRows; ++r)
						wv[r] = o0 + r < o_end
								? __ldg(reinterpret_cast<const float4 *>(
									  W + (size_t)(o0 + r) * width + k))
								: make_float4(0.f, 0.f, 0.f, 0.f);
					const float4 x0 = *reinterpret_cast<const float4 *>(a + k);
					const float4 x1 = *reinterpret_cast<const float4 *>(a + width + k);
#pragma unroll
					for (uint32_t r = 0; r < kDeltaRows; ++r) {
						z0[r] += dot4(wv[r], x0);
						z1[r] += dot4(wv[r], x1);
					}
				}
			} else {
				for (uint32_t k = lane; k < width; k += 32) {
					float wv[kDeltaRows];
#pragma unroll
					for (uint32_t r = 0; r < kDeltaRows; ++r)
						wv[r] = o0 + r < o_end
								? __ldg(W + (size_t)(o0 + r) * width + k)
								: 0.0f;
					const float x0 = a[k], x1 = a[width + k];
#pragma unroll
					for (uint32_t r = 0; r < kDeltaRows; ++r) {
						z0[r] = fmaf(wv[r], x0, z0[r]);
						z1[r] = fmaf(wv[r], x1, z1[r]);
					}
				}
			}
#pragma unroll
			for (uint32_t r = 0; r < kDeltaRows; ++r) {
				for (int off = 16; off > 0; off >>= 1) {
					z0[r] += __shfl_xor_sync(0xffffffffu, z0[r], off);
					z1[r] += __shfl_xor_sync(0xffffffffu, z1[r], off);
				}
				const uint32_t o = o0 + r;
				if (o < o_end && lane < 2 * kDeltaCluster) {
					const float bo = __ldg(bias + o);
					const bool second = lane >= kDeltaCluster;
					float *dst = cluster.map_shared_rank(b, lane % kDeltaCluster);
					dst[(second ? hidden : 0u) + o] =
						gelu((second ? z1[r] : z0[r]) + bo);
				}
			}
		}
		cluster.sync(); // the layer is complete in every CTA
		float *t = a;
		a = b;
		b = t;
		W = bias + hidden;
		width = hidden;
	}
	// output unit: W [1][hidden]; its bias cancels in the difference
	if (rank == 0 && warp == 0) {
		float y0 = 0.0f, y1 = 0.0f;
		for (uint32_t k = lane; k < hidden; k += 32) {
			const float wk = __ldg(W + k);
			y0 = fmaf(wk, a[k], y0);
			y1 = fmaf(wk, a[hidden + k], y1);
		}
		for (int off = 16; off > 0; off >>= 1) {
			y0 += __shfl_xor_sync(0xffffffffu, y0, off);
			y1 += __shfl_xor_sync(0xffffffffu, y1, off);
		}
		if (lane == 0) {
			*(volatile float *)out = y0 - y1;
			__threadfence_system();
		}
	}
}

} // namespace

Mlp::Mlp(uint32_t in_dim, uint32_t hidden, uint64_t seed, int device)
    : in_(in_dim), hidden_(hidden), device_(device)
{
	if (in_dim < 1 || in_dim > hidden || hidden < 32 || hidden > 1024 ||
	    hidden % 32 != 0)
		throw Error(B3G_ERR_INVALID_ARGUMENT,
			    "surrogate: 1 <= inputs <= 256, hidden a multiple of 32 "
			    "in 32..1024");
	check_cuda(cudaSetDevice(device), "cudaSetDevice");
	dims_[0] = in_dim;
	dims_[1] = dims_[2] = dims_[3] = hidden;
	dims_[4] = 1;
	uint32_t off = 0;
	for (uint32_t l = 0; l < kLayers; ++l) {
		w_off_[l] = off;
		off += dims_[l + 1] * dims_[l];
		b_off_[l] = off;
		off += dims_[l + 1];
	}
	n_params_ = off;
	// uniform(-1/sqrt(fan_in), 1/sqrt(fan_in)) weights, zero biases
	std::vector<float> p(n_params_, 0.0f);
	std::mt19937_64 gen(seed);
	for (uint32_t l = 0; l < kLayers; ++l) {
		const float r = 1.0f / std::sqrt(static_cast<float>(dims_[l]));
		std::uniform_real_distribution<float> u(-r, r);
		for (uint32_t k = 0; k < dims_[l + 1] * dims_[l]; ++k)
			p[w_off_[l] + k] = u(gen);
	}
	check_cuda(cudaStreamCreateWithFlags(&stream_, cudaStreamNonBlocking), "stream");
	const size_t bytes = sizeof(float) * n_params_;
	check_cuda(cudaMalloc(&d_params_, bytes), "surrogate params");
	check_cuda(cudaMalloc(&d_grad_, bytes), "surrogate grads");
	check_cuda(cudaMalloc(&d_m_, bytes), "adam m");
	check_cuda(cudaMalloc(&d_v_, bytes), "adam v");
	check_cuda(cudaMemcpy(d_params_, p.data(), bytes, cudaMemcpyHostToDevice), "params");
	check_cuda(cudaMemset(d_m_, 0, bytes), "adam m");
	check_cuda(cudaMemset(d_v_, 0, bytes), "adam v");
	// inference pairs and results in host-mapped memory: no copies, no
	// stream synchronisation per screening; results [kDeltaMax] first,
	// then the pairs [kDeltaMax][2 in]
	check_cuda(cudaHostAlloc((void **)&h_pair_,
				 sizeof(float) * kDeltaMax * (1 + 2 * in_),
				 cudaHostAllocMapped),
		   "mapped pairs");
	check_cuda(cudaHostGetDevicePointer((void **)&d_pair_, h_pair_, 0), "mapped pair");
}

Mlp::~Mlp()
{
	cudaSetDevice(device_);
	if (stream_)
		cudaStreamSynchronize(stream_);
	cudaFree(d_params_);
	cudaFree(d_grad_);
	cudaFree(d_m_);
	cudaFree(d_v_);
	free_batch();
	cudaFreeHost(h_pair_);
	for (InferCtx &c : extra_) {
		cudaStreamSynchronize(c.stream);
		cudaStreamDestroy(c.stream);
		cudaFreeHost(c.h);
	}
	if (stream_)
		cudaStreamDestroy(stream_);
}

void Mlp::free_batch()
{
	cudaFree(d_batch_);
	d_batch_ = nullptr;
	for (uint32_t l = 0; l + 1 < kLayers; ++l)
		d_z_[l] = d_a_[l] = d_dz_[l] = nullptr;
	d_x_ = d_y_ = d_delta_ = d_dys_ = d_loss_ = d_head_ = d_part_ = nullptr;
	d_tickets_ = nullptr;
	cap_ = grads_cap_ = parts_cap_ = 0;
}

namespace {
uint32_t dw_tiles(uint32_t O, uint32_t I)
{
	return ((O + kTm - 1) / kTm) * ((I + kTn - 1) / kTn);
}
uint32_t dw_split_rows(uint32_t rows)
{
	const uint32_t share = (rows + kSplits - 1) / kSplits;
	return std::max(kSplitRows, (share + kTk - 1) / kTk * kTk);
}
uint32_t head_blocks(uint32_t rows) // rows: two a pair
{
	return (rows / 2 + kHeadPairs - 1) / kHeadPairs;
}
} // namespace

// Workspaces for `rows` rows: what a gradient needs only for gradients, and the
// partial tiles of split weight gradients only where its rows are split (they
// are the largest: 4.3 MB for 256 units, 68 for 1,024).  An allocation beyond a
// megabyte is mapped on its own: a first forward pass of 64 rows and 256 units
// took 161 us with everything (95 as a dozen allocations), 84 now.
void Mlp::ensure_batch(uint32_t rows, bool gradient)
{
	uint32_t grads = gradient ? rows : 0u;
	uint32_t parts = grads > kSplitRows ? std::min(kSplits, (rows + kSplitRows - 1) / kSplitRows)
					    : 0u;
	if (rows <= cap_ && grads <= grads_cap_ && parts <= parts_cap_)
		return;
	rows = std::max(rows, cap_);
	grads = std::max(grads, grads_cap_);
	parts = std::max(parts, parts_cap_);
	check_cuda(cudaStreamSynchronize(stream_), "sync");
	free_batch();
	// one allocation, carved up (sixteen calls were half of the first
	// evaluation's time at small sizes)
	const uint32_t tiles = dw_tiles(hidden_, hidden_);
	size_t bytes = 0;
	auto carve = [&](auto *&p, size_t count) {
		const size_t at = bytes;
		bytes += (count * sizeof(*p) + 255) & ~(size_t)255;
		if (d_batch_)
			p = reinterpret_cast<std::decay_t<decltype(p)>>(d_batch_ + at);
	};
	auto all = [&] {
		bytes = 0;
		carve(d_tickets_, tiles + 1);
		carve(d_x_, (size_t)rows * in_);
		for (uint32_t l = 0; l + 1 < kLayers; ++l) {
			const size_t count = (size_t)rows * dims_[l + 1];
			carve(d_z_[l], count);
			carve(d_a_[l], count);
			carve(d_dz_[l], (size_t)grads * dims_[l + 1]);
		}
		carve(d_y_, rows);
		carve(d_delta_, grads);
		carve(d_dys_, grads);
		carve(d_loss_, 1);
		carve(d_head_, head_blocks(grads)); // the head kernel's block losses
		carve(d_part_, (size_t)tiles * parts * (kTm * kTn + kTm));
	};
	all();
	check_cuda(cudaMalloc(&d_batch_, bytes), "batch workspace");
	all();
	check_cuda(cudaMemsetAsync(d_tickets_, 0, sizeof(unsigned) * (tiles + 1), stream_),
		   "zero tickets");
	cap_ = rows;
	grads_cap_ = grads;
	parts_cap_ = parts;
}

// d_x_ rows through the hidden layers (z and a of each).
void Mlp::forward_device(uint32_t rows)
{
	const float *in = d_x_;
	for (uint32_t l = 0; l + 1 < kLayers; ++l) {
		const uint32_t I = dims_[l], O = dims_[l + 1];
		mlp_forward_kernel<<<dim3((O + kTn - 1) / kTn, (rows + kTm - 1) / kTm), kTt, 0,
				     stream_>>>(in, d_params_ + w_off_[l], d_params_ + b_off_[l],
						d_z_[l], d_a_[l], rows, O, I);
		in = d_a_[l];
	}
	check_cuda(cudaGetLastError(), "surrogate forward");
}

// Pair objective of `n` pairs (2 n rows in d_a_, d_delta_) and its gradient:
// d_loss_, d_grad_.
void Mlp::backward_device(uint32_t n)
{
	const uint32_t rows = 2 * n, H = hidden_, top = kLayers - 2;
	const uint32_t hb = head_blocks(rows);
	mlp_head_kernel<<<hb, 32 * kHeadPairs, sizeof(float) * (2 * kHeadPairs + 1) * head_row(H),
			  stream_>>>(d_a_[top], d_z_[top], d_params_ + w_off_[kLayers - 1], d_delta_,
				     d_dz_[top], d_dys_, d_head_, d_loss_,
				     d_tickets_ + dw_tiles(H, H), n, H);
	for (int l = (int)top; l >= 0; --l) {
		MlpBackward p{};
		p.rows = rows;
		p.O = dims_[l + 1];
		p.I = dims_[l];
		p.dz = d_dz_[l];
		p.a = l == 0 ? d_x_ : d_a_[l - 1];
		p.W = d_params_ + w_off_[l];
		p.dW = d_grad_ + w_off_[l];
		p.db = d_grad_ + b_off_[l];
		p.part = d_part_;
		p.tickets = d_tickets_;
		p.split_rows = dw_split_rows(rows);
		p.splits = (rows + p.split_rows - 1) / p.split_rows;
		p.dw_blocks = dw_tiles(p.O, p.I) * p.splits;
		if (l > 0) {
			p.z_below = d_z_[l - 1];
			p.dz_below = d_dz_[l - 1];
			p.da_blocks = ((rows + kTm - 1) / kTm) * ((p.I + kTn - 1) / kTn);
		}
		uint32_t blocks = p.dw_blocks + p.da_blocks;
		if (l == (int)top) {
			p.dys = d_dys_;
			p.a_out = d_a_[l];
			p.head_grad = d_grad_ + w_off_[kLayers - 1]; // weights, then the bias
			blocks += 2 * ((H + kChainCols - 1) / kChainCols);
		}
		mlp_backward_kernel<<<blocks, kTt, 0, stream_>>>(p);
	}
	check_cuda(cudaGetLastError(), "surrogate backward");
}

void Mlp::get_params(float *out)
{
	check_cuda(cudaStreamSynchronize(stream_), "sync");
	check_cuda(cudaMemcpy(out, d_params_, sizeof(float) * n_params_,
			      cudaMemcpyDeviceToHost),
		   "read params");
}

void Mlp::set_params(const float *in)
{
	check_cuda(cudaStreamSynchronize(stream_), "sync");
	check_cuda(cudaMemcpy(d_params_, in, sizeof(float) * n_params_,
			      cudaMemcpyHostToDevice),
		   "write params");
	check_cuda(cudaMemset(d_m_, 0, sizeof(float) * n_params_), "adam m");
	check_cuda(cudaMemset(d_v_, 0, sizeof(float) * n_params_), "adam v");
	adam_t_ = 0;
}

void Mlp::forward(const float *x, uint32_t n, float *out)
{
	check_cuda(cudaSetDevice(device_), "cudaSetDevice");
	ensure_batch(n, false);
	check_cuda(cudaMemcpyAsync(d_x_, x, sizeof(float) * n * in_,
				   cudaMemcpyHostToDevice, stream_),
		   "inputs");
	forward_device(n);
	mlp_out_kernel<<<(n + 7) / 8, 256, 0, stream_>>>(
		d_a_[kLayers - 2], d_params_ + w_off_[kLayers - 1], d_y_, n, hidden_);
	check_cuda(cudaGetLastError(), "surrogate output");
	check_cuda(cudaMemcpyAsync(out, d_y_, sizeof(float) * n,
				   cudaMemcpyDeviceToHost, stream_),
		   "outputs");
	check_cuda(cudaStreamSynchronize(stream_), "sync");
}

float Mlp::loss_grad(const float *x_new, const float *x_old,
		     const float *delta, uint32_t n, float *grad)
{
	check_cuda(cudaSetDevice(device_), "cudaSetDevice");
	ensure_batch(2 * n, true);
	check_cuda(cudaMemcpyAsync(d_x_, x_new, sizeof(float) * n * in_,
				   cudaMemcpyHostToDevice, stream_),
		   "inputs");
	check_cuda(cudaMemcpyAsync(d_x_ + (size_t)n * in_, x_old,
				   sizeof(float) * n * in_, cudaMemcpyHostToDevice,
				   stream_),
		   "inputs");
	check_cuda(cudaMemcpyAsync(d_delta_, delta, sizeof(float) * n,
				   cudaMemcpyHostToDevice, stream_),
		   "deltas");
	forward_device(2 * n);
	backward_device(n);
	float loss = 0.0f;
	check_cuda(cudaMemcpyAsync(&loss, d_loss_, sizeof(float),
				   cudaMemcpyDeviceToHost, stream_),
		   "loss");
	if (grad)
		check_cuda(cudaMemcpyAsync(grad, d_grad_, sizeof(float) * n_params_,
					   cudaMemcpyDeviceToHost, stream_),
			   "grads");
	check_cuda(cudaStreamSynchronize(stream_), "sync");
	return loss;
}

float Mlp::train(const float *x_new, const float *x_old, const float *delta,
		 uint32_t n, uint32_t epochs, uint32_t batch, float lr,
		 uint64_t seed)
{
	if (n < 1 || batch < 1)
		throw Error(B3G_ERR_INVALID_ARGUMENT, "empty training set");
	check_cuda(cudaSetDevice(device_), "cudaSetDevice");
	batch = std::min(batch, n);
	ensure_batch(2 * batch, true);
	// the whole data set on the device once: rows [x_new; x_old], deltas
	float *d_xn = nullptr, *d_xo = nullptr, *d_dl = nullptr;
	uint32_t *d_idx = nullptr, *h_idx = nullptr;
	check_cuda(cudaMalloc(&d_xn, sizeof(float) * n * in_), "train x_new");
	check_cuda(cudaMalloc(&d_xo, sizeof(float) * n * in_), "train x_old");
	check_cuda(cudaMalloc(&d_dl, sizeof(float) * n), "train deltas");
	check_cuda(cudaMalloc(&d_idx, sizeof(uint32_t) * batch), "indices");
	check_cuda(cudaHostAlloc((void **)&h_idx, sizeof(uint32_t) * batch,
				 cudaHostAllocDefault),
		   "pinned indices");
	check_cuda(cudaMemcpy(d_xn, x_new, sizeof(float) * n * in_, cudaMemcpyHostToDevice), "x_new");
	check_cuda(cudaMemcpy(d_xo, x_old, sizeof(float) * n * in_, cudaMemcpyHostToDevice), "x_old");
	check_cuda(cudaMemcpy(d_dl, delta, sizeof(float) * n, cudaMemcpyHostToDevice), "deltas");
	std::vector<uint32_t> order(n);
	std::iota(order.begin(), order.end(), 0u);
	std::mt19937_64 gen(seed);
	const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
	double epoch_loss = 0.0;
	for (uint32_t e = 0; e < epochs; ++e) {
		std::shuffle(order.begin(), order.end(), gen);
		epoch_loss = 0.0;
		uint32_t batches = 0;
		for (uint32_t s = 0; s + batch <= n; s += batch) {
			check_cuda(cudaStreamSynchronize(stream_), "sync");
			std::memcpy(h_idx, order.data() + s, sizeof(uint32_t) * batch);
			check_cuda(cudaMemcpyAsync(d_idx, h_idx, sizeof(uint32_t) * batch,
						   cudaMemcpyHostToDevice, stream_),
				   "indices");
			const uint32_t cnt = batch * in_;
			gather_rows_kernel<<<(cnt + 255) / 256, 256, 0, stream_>>>(
				d_xn, d_idx, d_x_, batch, in_);
			gather_rows_kernel<<<(cnt + 255) / 256, 256, 0, stream_>>>(
				d_xo, d_idx, d_x_ + (size_t)batch * in_, batch, in_);
			gather_rows_kernel<<<(batch + 255) / 256, 256, 0, stream_>>>(
				d_dl, d_idx, d_delta_, batch, 1);
			forward_device(2 * batch);
			backward_device(batch);
			++adam_t_;
			const float c1 = 1.0f - std::pow(b1, (float)adam_t_);
			const float c2 = 1.0f - std::pow(b2, (float)adam_t_);
			adam_kernel<<<(n_params_ + 255) / 256, 256, 0, stream_>>>(
				d_params_, d_grad_, d_m_, d_v_, n_params_, lr, b1, b2,
				c1, c2, eps);
			float loss = 0.0f;
			check_cuda(cudaMemcpyAsync(&loss, d_loss_, sizeof(float),
						   cudaMemcpyDeviceToHost, stream_),
				   "loss");
			check_cuda(cudaStreamSynchronize(stream_), "sync");
			epoch_loss += loss;
			++batches;
		}
		epoch_loss /= std::max(1u, batches);
	}
	cudaFree(d_xn);
	cudaFree(d_xo);
	cudaFree(d_dl);
	cudaFree(d_idx);
	cudaFreeHost(h_idx);
	check_cuda(cudaGetLastError(), "training");
	return static_cast<float>(epoch_loss);
}

namespace {
// a NaN payload the kernel never writes
constexpr uint32_t kDeltaSentinel = 0x7fb3a5e1u;
} // namespace

float Mlp::delta(const float *x_new, const float *x_old)
{
	float out;
	deltas(x_new, x_old, 1, &out);
	return out;
}

void Mlp::ensure_contexts(uint32_t n)
{
	check_cuda(cudaSetDevice(device_), "cudaSetDevice");
	int least = 0, greatest = 0;
	check_cuda(cudaDeviceGetStreamPriorityRange(&least, &greatest), "stream priorities");
	while (extra_.size() + 1 < n) {
		InferCtx c{};
		check_cuda(cudaStreamCreateWithPriority(&c.stream, cudaStreamNonBlocking,
							 greatest),
			   "surrogate stream");
		check_cuda(cudaHostAlloc((void **)&c.h, sizeof(float) * kDeltaMax * (1 + 2 * in_),
					 cudaHostAllocMapped),
			   "mapped pairs");
		check_cuda(cudaHostGetDevicePointer((void **)&c.d, c.h, 0), "mapped pairs");
		extra_.push_back(c);
	}
}

void Mlp::deltas(const float *x_new, const float *x_old, uint32_t count, float *out)
{
	deltas(0, x_new, x_old, count, out);
}

void Mlp::deltas(uint32_t ctx, const float *x_new, const float *x_old, uint32_t count,
		 float *out)
{
	if (count == 0)
		return;
	if (count > kDeltaMax)
		throw Error(B3G_ERR_INVALID_ARGUMENT, "too many surrogate pairs at once");
	if (ctx > extra_.size())
		throw Error(B3G_ERR_INVALID_ARGUMENT, "no such surrogate context");
	float *const h_pair = ctx ? extra_[ctx - 1].h : h_pair_;
	float *const d_pair = ctx ? extra_[ctx - 1].d : d_pair_;
	const cudaStream_t stream = ctx ? extra_[ctx - 1].stream : stream_;
	volatile uint32_t *words = reinterpret_cast<volatile uint32_t *>(h_pair);
	float *pairs = h_pair + kDeltaMax;
	const uint32_t stride = 2 * in_;
	for (uint32_t k = 0; k < count; ++k) {
		std::memcpy(pairs + (size_t)k * stride, x_new + (size_t)k * in_,
			    sizeof(float) * in_);
		std::memcpy(pairs + (size_t)k * stride + in_, x_old + (size_t)k * in_,
			    sizeof(float) * in_);
		words[k] = kDeltaSentinel;
	}
	std::atomic_thread_fence(std::memory_order_seq_cst);
	const size_t smem = sizeof(float) * 2 * (std::max(hidden_, in_) + hidden_);
	mlp_delta_kernel<<<kDeltaCluster * count, 256, smem, stream>>>(
		d_params_, d_pair + kDeltaMax, d_pair, in_, hidden_, stride);
	check_cuda(cudaGetLastError(), "surrogate inference");
	// poll the mapped words; every 64 polls ask the stream, so that an
	// error surfaces and a finished kernel that wrote nothing ends the wait
	uint32_t k = 0;
	for (uint32_t poll = 1; k < count; ++poll) {
		uint32_t bits = words[k];
		if (bits != kDeltaSentinel) {
			std::memcpy(out + k, &bits, sizeof(float));
			++k;
			continue;
		}
		if ((poll & 63u) == 0) {
			const cudaError_t e = cudaStreamQuery(stream);
			if (e == cudaSuccess) {
				for (; k < count; ++k) {
					bits = words[k];
					if (bits == kDeltaSentinel)
						throw Error(B3G_ERR_CUDA,
							    "surrogate inference finished without a result");
					std::memcpy(out + k, &bits, sizeof(float));
				}
				return;
			}
			if (e != cudaErrorNotReady)
				check_cuda(e, "surrogate inference");
		}
	}
}

} // namespace b3g
