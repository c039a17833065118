// Gradient::calculate (gradient.cpp:20-75), the padded pixel image read by
// the PatchMatch distance, mask compaction and small reductions.
#include "nli_device.cuh"

namespace nli {

// Forward differences per channel, 0 on the last column / row; output has
// 2C interleaved channels [gx_0, gy_0, gx_1, gy_1, ...].  One thread per
// pixel and channel; consecutive threads touch consecutive addresses.
__global__ void k_gradient(const float *__restrict__ img, int W, int H, int C, float *__restrict__ grad)
{
	gradient_span(img, W, H, C, grad, blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x);
}

void launch_gradient(cudaStream_t s, const float *img, int W, int H, int C, float *grad)
{
	const int n = W * H * C;
	const int block = 256, grid = (n + block - 1) / block;
	k_gradient<<<grid, block, 0, s>>>(img, W, H, C, grad);
	NLI_CHECK_LAUNCH();
}

// Pixels read by the PatchMatch distance: one float4 per pixel (channels
// 0..C-1, the rest zero) over (W + 1) x (H + 1), the extra column and row
// repeating the last ones so that forward differences there are exactly 0.
__global__ void k_pad4(const float *__restrict__ img, int W, int H, int C, float4 *__restrict__ out)
{
	next_launch_may_start();
	previous_launch_done();
	pad4_span(img, W, H, C, out, blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x);
}

void launch_pad4(cudaStream_t s, const float *img, int W, int H, int C, float4 *out)
{
	const int n = (W + 1) * (H + 1);
	const int block = 256, grid = (n + block - 1) / block;
	launch_early(s, grid, block, 0, k_pad4, img, W, H, C, out);
	NLI_CHECK_LAUNCH();
}

// ---------------------------------------------------------- compaction
// Raster-order list of the set pixels of a mask: per-tile counts, then per-tile
// ordered writes, each block adding up the counts before its own.  (As three
// launches, with one block scanning in between and a copy of the total to the
// host, it took 14 us, nearly all of it latency, 7 of it the scan's serial part: a
// PatchMatch call on 64 x 48 goes from 231 to 220 us, a Poisson update of
// 512 x 512 from 317 to 301.)  Above 2 M pixels, more than two counts a
// thread, the scan stays.
constexpr int kTile = 1024;
constexpr int kPrefixTiles = 2048;

__global__ void k_count(const uint8_t *__restrict__ mask, int n, int *__restrict__ counts)
{
	next_launch_may_start();
	previous_launch_done();
	__shared__ int s[32];
	const int base = blockIdx.x * kTile;
	int c = 0;
	for (int i = threadIdx.x; i < kTile; i += blockDim.x) {
		const int p = base + i;
		c += (p < n && mask[p]) ? 1 : 0;
	}
	for (int o = 16; o > 0; o >>= 1) c += __shfl_down_sync(0xffffffffu, c, o);
	if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = c;
	__syncthreads();
	if (threadIdx.x == 0) {
		int t = 0;
		for (int w = 0; w < (int)(blockDim.x >> 5); w++) t += s[w];
		counts[blockIdx.x] = t;
	}
}

// Exclusive sum of one value per thread over a block of 1024; `sums` (33 words)
// keeps the total in its last word.
__device__ __forceinline__ int block_exclusive(int v, int *sums)
{
	const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
	int incl = v;
	for (int o = 1; o < 32; o <<= 1) {
		const int t = __shfl_up_sync(0xffffffffu, incl, o);
		if (lane >= o) incl += t;
	}
	if (lane == 31) sums[wid] = incl;
	__syncthreads();
	if (wid == 0) {
		const int own = sums[lane];
		int all = own;
		for (int o = 1; o < 32; o <<= 1) {
			const int t = __shfl_up_sync(0xffffffffu, all, o);
			if (lane >= o) all += t;
		}
		sums[lane] = all - own;
		if (lane == 31) sums[32] = all;
	}
	__syncthreads();
	return sums[wid] + incl - v;
}

// Single block: exclusive scan of the tile counts, sequential chunks per thread.
__global__ void __launch_bounds__(1024) k_scan(int *__restrict__ counts, int tiles)
{
	__shared__ int sums[33];
	const int per = (tiles + 1023) / 1024;
	const int b = threadIdx.x * per, e = min(b + per, tiles);
	int s = 0;
	for (int i = b; i < e; i++) s += counts[i];
	int run = block_exclusive(s, sums);
	for (int i = b; i < e; i++) {
		const int v = counts[i];
		counts[i] = run;
		run += v;
	}
}

// 1024 threads, one pixel each: block-wide ordered scan of the flags.  SCANNED:
// `counts` are the exclusive sums, else the tiles' own.  The last block
// writes the total, to pinned memory.
template <bool SCANNED>
__global__ void __launch_bounds__(kTile)
    k_write(const uint8_t *__restrict__ mask, int n, const int *__restrict__ counts, int32_t *__restrict__ list,
            int *__restrict__ total)
{
	next_launch_may_start();
	previous_launch_done();
	__shared__ int sums[33], before;
	const int p = blockIdx.x * kTile + threadIdx.x;
	const int f = (p < n && mask[p]) ? 1 : 0;
	if (threadIdx.x == 0) before = SCANNED ? counts[blockIdx.x] : 0;
	if (!SCANNED) {
		int c = 0;
		for (int i = threadIdx.x; i < (int)blockIdx.x; i += kTile) c += counts[i];
		c = __reduce_add_sync(0xffffffffu, c);
		__syncthreads();
		if ((threadIdx.x & 31) == 0 && c) atomicAdd(&before, c);
	}
	const int at = block_exclusive(f, sums);  // its barriers order `before`
	if (f) list[before + at] = p;
	if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) *total = before + sums[32];
}

int compact_mask(nli_ctx *ctx, const uint8_t *mask, int W, int H, int32_t *list, const char *tag)
{
	const int n = W * H;
	const int tiles = (n + kTile - 1) / kTile;
	int *counts = ctx->buf<int>(std::string("compact.counts.") + tag, tiles);
	int *total = (int *)ctx->host_pinned;
	launch_early(ctx->stream, tiles, 256, 0, k_count, mask, n, counts);
	NLI_CHECK_LAUNCH();
	if (tiles > kPrefixTiles) {
		k_scan<<<1, 1024, 0, ctx->stream>>>(counts, tiles);
		NLI_CHECK_LAUNCH();
		launch_early(ctx->stream, tiles, kTile, 0, k_write<true>, mask, n, counts, list, total);
	} else {
		launch_early(ctx->stream, tiles, kTile, 0, k_write<false>, mask, n, counts, list, total);
	}
	NLI_CHECK_LAUNCH();
	NLI_CUDA(cudaStreamSynchronize(ctx->stream));
	return *(volatile int *)total;
}

// Sum of n doubles in a fixed order (one block), for repeatable totals.
__global__ void k_sum_partials(const double *__restrict__ partials, int n, double *__restrict__ out)
{
	next_launch_may_start();
	previous_launch_done();
	__shared__ double s[32];
	double v = 0.0;
	for (int i = threadIdx.x; i < n; i += blockDim.x) v += partials[i];
	v = block_sum<1024>(v, s);
	if (threadIdx.x == 0) *out = v;
}

void launch_sum_partials(cudaStream_t s, const double *partials, int n, double *out)
{
	launch_early(s, 1, 1024, 0, k_sum_partials, partials, n, out);
	NLI_CHECK_LAUNCH();
}

}  // namespace nli
