// PatchMatch's entry points: buffers, tables and launches around the sweep
// kernels of pm_kernels.cuh, which pm_*.cu instantiate.
#include <cmath>

#include "pm_kernels.cuh"

namespace nli {

// ------------------------------------------------------ bound tables
// Factors of the patch weights along x and y and the slopes' weights: f_1 =
// (x - mean x) / sigma_x under the weights, f_2 likewise in y (0 for a side of
// one tap, whose slope says nothing).
static void patch_factors(PmFactors &f, const DistArgs &a)
{
	std::memset(&f, 0, sizeof(f));
	f.px = a.px;
	f.py = a.py;
	f.rx = a.rx;
	f.ry = a.ry;
	auto axis = [](const double *w, int n, float *ow, float *of) {
		double mean = 0.0, var = 0.0;
		for (int i = 0; i < n; i++) mean += w[i] * i;
		for (int i = 0; i < n; i++) var += w[i] * (i - mean) * (i - mean);
		for (int i = 0; i < n; i++) {
			ow[i] = (float)w[i];
			of[i] = var > 1e-9 ? (float)(w[i] * (i - mean) / std::sqrt(var)) : 0.f;
		}
	};
	double wx[NLI_MAX_PATCH] = {}, wy[NLI_MAX_PATCH] = {};
	for (int y = 0; y < a.py; y++)
		for (int x = 0; x < a.px; x++) {
			wx[x] += a.weights[y * a.px + x];
			wy[y] += a.weights[y * a.px + x];
		}
	axis(wx, a.px, f.wx, f.fx);
	axis(wy, a.py, f.wy, f.fy);
}

// Whether the L2 kinds' bound uses the slopes for an image of nt target points:
// the terms it bounds have non-negative factors, and the call is one whose
// points come in groups (pm_group) -- there a candidate less is a part of a
// round less, while a small call waits longer for the second test than for
// the evaluations it saves (64 x 48: 296 us without, 317 with; 130 x 81: 355
// and 373; 512 x 512: 1466 and 1382).  By the image's own size, so that a
// batch tests as the image alone does.
static int bound_slopes(const nli_distance_params &d, int nt, int num_sms)
{
	if (nt < 48 * num_sms) return 0;
	auto share = [](float v) { return v >= 0.f && v <= 1.f; };
	if (d.kind == NLI_DIST_L1_NORM) return 0;
	if (d.kind == NLI_DIST_L2_NORM) return 1;
	return share(d.lambda) && (d.kind != NLI_DIST_L2_RGBD || share(d.lambda_d));
}

int pm_moment_tables(const nli_ctx *ctx, const nli_distance_params &d, int nt)
{
	if (!ctx->tune_pm_bound) return 0;
	if (ctx->tune_pm_bound == 2 && d.kind != NLI_DIST_L1_NORM) return 6;
	return bound_slopes(d, nt, ctx->num_sms) ? 3 : 1;
}

// Means and slopes of every position of the padded (W + 1) x (H + 1) grid
// (window clamped to the grid), and the largest absolute pixel value (atomicMax
// on the float bits of non-negative values).  The weights are a product of
// factors, so a tile of kMomW x kMomH positions sums along x (w and w f_1)
// over its rows and the window's, then along y: 2 x 9 + 3 x 9 products per
// position instead of 3 x 81, every pixel read about 2.7 times instead of
// 81.  The one-pass form took 25.4 us for the means alone at 512 x 512 (bound
// by the L1 data pipe), this takes 13.1 us for means and slopes (15 MB written:
// 1.2 TB/s); 64 x 48: 8.9 and 4.8 us.
constexpr int kMomW = 32, kMomH = 8;

__device__ __forceinline__ void moments_tile(const PmFactors &f, const float4 *__restrict__ pad, int W, int H,
                                             float4 *__restrict__ mom, unsigned *vmax, int slopes, int tile)
{
	__shared__ float4 s_in[kMomH + NLI_MAX_PATCH - 1][kMomW + NLI_MAX_PATCH - 1];
	__shared__ float4 s_w[kMomH + NLI_MAX_PATCH - 1][kMomW], s_f[kMomH + NLI_MAX_PATCH - 1][kMomW];
	const int Wp = W + 1, tiles_x = (Wp + kMomW - 1) / kMomW;
	const int x0 = (tile % tiles_x) * kMomW, y0 = (tile / tiles_x) * kMomH;
	const int cols = kMomW + f.px - 1, rows = kMomH + f.py - 1;
	for (int e = threadIdx.x; e < rows * cols; e += blockDim.x) {
		const int r = e / cols, c = e - r * cols;
		const int y = min(max(y0 - f.ry + r, 0), H), x = min(max(x0 - f.rx + c, 0), W);
		s_in[r][c] = __ldg(pad + (size_t)y * Wp + x);
	}
	__syncthreads();
	const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
	for (int e = threadIdx.x; e < rows * kMomW; e += blockDim.x) {
		const int r = e / kMomW, c = e - r * kMomW;
		float4 a = zero, b = zero;
		for (int i = 0; i < f.px; i++) {
			const float4 v = s_in[r][c + i];
			a = f4_fma(f.wx[i], v, a);
			b = f4_fma(f.fx[i], v, b);
		}
		s_w[r][c] = a;
		s_f[r][c] = b;
	}
	__syncthreads();
	const int c = threadIdx.x % kMomW, r = threadIdx.x / kMomW;
	const int x = x0 + c, y = y0 + r;
	float vm = 0.f;
	if (x <= W && y <= H) {
		float4 m = zero, sx = zero, sy = zero;
		for (int j = 0; j < f.py; j++) {
			const float4 a = s_w[r + j][c];
			m = f4_fma(f.wy[j], a, m);
			sx = f4_fma(f.wy[j], s_f[r + j][c], sx);
			sy = f4_fma(f.fy[j], a, sy);
		}
		const size_t i = (size_t)y * Wp + x, n = (size_t)Wp * (H + 1);
		mom[i] = m;
		if (slopes) {
			mom[n + 2 * i] = sx;
			mom[n + 2 * i + 1] = sy;
		}
		const float4 v = s_in[r + f.ry][c + f.rx];
		vm = fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w)));
	}
	for (int o = 16; o > 0; o >>= 1) vm = fmaxf(vm, __shfl_xor_sync(kFull, vm, o));
	if ((threadIdx.x & 31) == 0 && vm > 0.f) atomicMax(vmax, __float_as_uint(vm));
}

static int moment_tiles(int W, int H) { return ((W + 1 + kMomW - 1) / kMomW) * ((H + 1 + kMomH - 1) / kMomH); }

__global__ void __launch_bounds__(kMomW * kMomH)
    k_pm_moments(const __grid_constant__ PmFactors f, const float4 *__restrict__ pad, int W, int H,
                 float4 *__restrict__ mom, unsigned *vmax, int slopes)
{
	next_launch_may_start();
	previous_launch_done();
	moments_tile(f, pad, W, H, mom, vmax, slopes, blockIdx.x);
}

// The weighted standard deviations of the image and of its forward
// differences in x and in y (NLI_TUNE_PM_BOUND 2), tables 3 to 5 of n = (W +
// 1)(H + 1) float4: sqrt(sum_k w_k (v_k - mean)^2) from a second, centred pass.
__device__ __forceinline__ void deviations_span(const DistArgs &a, const float4 *__restrict__ pad, int W, int H,
                                                float4 *__restrict__ mom, int first, int stride)
{
	const int Wp = W + 1, n = Wp * (H + 1);
	const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
	for (int i = first; i < n; i += stride) {
		const int y = i / Wp, x = i - y * Wp;
		float4 mean[3] = {zero, zero, zero}, s[3] = {zero, zero, zero};
		for (int pass = 0; pass < 2; pass++)
			for (int dy = 0; dy < a.py; dy++) {
				const int yy = min(max(y - a.ry + dy, 0), H);
				const float4 *row = pad + (size_t)yy * Wp, *below = pad + (size_t)min(yy + 1, H) * Wp;
				for (int dx = 0; dx < a.px; dx++) {
					const int xx = min(max(x - a.rx + dx, 0), W);
					const float4 v = __ldg(row + xx);
					const float w = a.weights[dy * a.px + dx];
					const float4 d[3] = {v, f4_sub(__ldg(row + min(xx + 1, W)), v), f4_sub(__ldg(below + xx), v)};
#pragma unroll
					for (int k = 0; k < 3; k++) {
						if (pass == 0)
							mean[k] = f4_fma(w, d[k], mean[k]);
						else
							s[k] = f4_wsq(w, f4_sub(d[k], mean[k]), s[k]);
					}
				}
			}
#pragma unroll
		for (int k = 0; k < 3; k++) mom[(size_t)(3 + k) * n + i] = f4_sqrt(s[k]);
	}
}

__global__ void k_pm_deviations(DistArgs a, const float4 *__restrict__ pad, int W, int H, float4 *__restrict__ mom)
{
	deviations_span(a, pad, W, H, mom, blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x);
}

// Also advances the context's PatchMatch call index when `calls` is set.
__global__ void k_fill_nnf(int2 *__restrict__ nnf, float *__restrict__ dist, int n, unsigned long long *calls)
{
	next_launch_may_start();
	previous_launch_done();
	if (calls && blockIdx.x == 0 && threadIdx.x == 0) *calls += 1ull;
	for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
		nnf[i] = make_int2(-1, -1);
		if (dist) dist[i] = FLT_MAX;
	}
}

__global__ void k_copy_targets(const int32_t *__restrict__ tlist, int nt, const int2 *__restrict__ nnf_src,
                               const float *__restrict__ dist_src, int2 *__restrict__ nnf_dst,
                               float *__restrict__ dist_dst)
{
	next_launch_may_start();
	previous_launch_done();
	const int i = blockIdx.x * blockDim.x + threadIdx.x;
	if (i >= nt) return;
	const int pix = tlist[i];
	if (nnf_dst) nnf_dst[pix] = nnf_src[pix];
	if (dist_dst) dist_dst[pix] = dist_src[pix];
}

__global__ void k_energy(const int32_t *__restrict__ tlist, int nt, const float *__restrict__ dist,
                         double *__restrict__ partials)
{
	next_launch_may_start();
	previous_launch_done();
	__shared__ double s[32];
	double v = 0.0;
	for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nt; i += gridDim.x * blockDim.x) {
		const float d = dist[tlist[i]];
		if (d < FLT_MAX) v += (double)d;
	}
	v = block_sum<256>(v, s);
	if (threadIdx.x == 0) partials[blockIdx.x] = v;
}

// cuTensorMapEncodeTiled through the runtime's driver entry point (no
// link against the driver library); null when the driver does not have it.
typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_tiled()
{
	static const EncodeTiledFn fn = [] {
		void *f = nullptr;
		cudaDriverEntryPointQueryResult q = cudaDriverEntryPointSymbolNotFound;
		if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &f, 12000, cudaEnableDefault, &q) !=
		        cudaSuccess ||
		    q != cudaDriverEntryPointSuccess) {
			(void)cudaGetLastError();
			return static_cast<EncodeTiledFn>(nullptr);
		}
		return reinterpret_cast<EncodeTiledFn>(f);
	}();
	return fn;
}

// The padded source as a 2-D float tensor (4 * sWp floats by sH + 1 rows)
// with a box of one candidate window (4 * L floats by rows).  False when it
// cannot be encoded; the caller then reads the windows with plain loads.
bool encode_source_map(const PmArgs &p, CUtensorMap *map)
{
	const EncodeTiledFn enc = encode_tiled();
	if (!enc) return false;
	if ((reinterpret_cast<uintptr_t>(p.src) & 15) != 0 || 4 * p.L > 256 || p.rows > 256) return false;
	const cuuint64_t dim[2] = {(cuuint64_t)4 * p.sWp, (cuuint64_t)p.sH + 1};
	const cuuint64_t stride[1] = {(cuuint64_t)p.sWp * sizeof(float4)};
	const cuuint32_t box[2] = {(cuuint32_t)(4 * p.L), (cuuint32_t)p.rows};
	const cuuint32_t estride[2] = {1, 1};
	return enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float4 *>(p.src), dim, stride, box, estride,
	           CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
	           CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

void sweep_energy(cudaStream_t s, const PmArgs &p, const float *dist, const PmMetrics &m, int sweep)
{
	launch_early(s, m.partial_blocks, 256, 0, k_energy, p.tlist, p.nt, dist, m.partials);
	NLI_CHECK_LAUNCH();
	launch_sum_partials(s, m.partials, m.partial_blocks, m.energy + sweep);
}

// The padded float4 pixels of every active image (k_pad4 per image); the
// largest-value word of its patch means is cleared.
__global__ void k_pad4_batch(const __grid_constant__ PmBatchArgs B, int C)
{
	const int t = blockIdx.y;
	const PmBatchTask &T = B.t[t];
	if (!batch_on(B.active, T.flag)) return;
	if (T.p.vmax && blockIdx.x == 0 && threadIdx.x == 0) *const_cast<unsigned *>(T.p.vmax) = 0u;
	pad4_span(T.img, T.p.sW, T.p.sH, C, const_cast<float4 *>(T.p.src), blockIdx.x * blockDim.x + threadIdx.x,
	          gridDim.x * blockDim.x);
}

// k_pm_moments and k_pm_deviations per active image.
__global__ void __launch_bounds__(kMomW * kMomH)
    k_pm_moments_batch(const __grid_constant__ PmFactors f, const __grid_constant__ PmBatchArgs B)
{
	const int t = blockIdx.y;
	const PmBatchTask &T = B.t[t];
	if (!batch_on(B.active, T.flag) || (int)blockIdx.x >= T.moment_tiles) return;
	moments_tile(f, T.p.src, T.p.sW, T.p.sH, const_cast<float4 *>(T.p.smom), const_cast<unsigned *>(T.p.vmax),
	             T.p.slopes, blockIdx.x);
}

__global__ void k_pm_deviations_batch(DistArgs a, const __grid_constant__ PmBatchArgs B)
{
	const int t = blockIdx.y;
	const PmBatchTask &T = B.t[t];
	if (!batch_on(B.active, T.flag)) return;
	deviations_span(a, T.p.src, T.p.sW, T.p.sH, const_cast<float4 *>(T.p.smom),
	                blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x);
}

// k_fill_nnf per active image: the result field to "none", and the image's
// call index advanced when it has target points.
__global__ void k_fill_nnf_batch(const __grid_constant__ PmBatchArgs B)
{
	const int t = blockIdx.y;
	const PmBatchTask &T = B.t[t];
	if (!batch_on(B.active, T.flag)) return;
	if (T.p.nt > 0 && blockIdx.x == 0 && threadIdx.x == 0) *const_cast<unsigned long long *>(T.p.calls) += 1ull;
	const int n = T.p.tW * T.p.tH;
	for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
		T.nnf_x[i] = make_int2(-1, -1);
}

// After an odd number of sweeps the field is in the second buffer: copy
// the target points back (k_copy_targets per active image).
__global__ void k_copy_targets_batch(const __grid_constant__ PmBatchArgs B)
{
	const int t = blockIdx.y;
	const PmBatchTask &T = B.t[t];
	if (!batch_on(B.active, T.flag)) return;
	for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < T.p.nt; i += gridDim.x * blockDim.x) {
		const int pix = T.p.tlist[i];
		T.nnf_x[pix] = T.io[0].nnf_out[pix];
	}
}

void patchmatch_batch_run(nli_ctx *ctx, const nli_distance_params &dp, const nli_patchmatch_params &pm, int C, int n,
                          const PmBatchItem *items, const int *active)
{
	NLI_REQUIRE(n >= 1 && n <= kBatchMax, NLI_E_INVALID, "batched PatchMatch takes 1 to 64 images");
	DistArgs a;
	fill_dist_args(a, dp, C);
	const bool grad = dp.kind == NLI_DIST_L2_COMBINED || dp.kind == NLI_DIST_L2_RGBD;
	PmBatchArgs B;
	std::memset(&B, 0, sizeof(B));
	B.n = n;
	B.active = active;
	B.tile = ctx->tune_pm_tile;
	int maxpix = 0, maxpad = 0, maxnt = 0;
	long long total = 0;  // target points of all images
	int maxtiles = 0;
	int widest = 0;       // the largest random-search window (as unsigned)
	for (int i = 0; i < n; i++) {
		const PmBatchItem &it = items[i];
		NLI_REQUIRE(it.W < 32768 && it.H < 32768, NLI_E_UNSUPPORTED, "PatchMatch source sides must be below 32768");
		PmBatchTask &T = B.t[i];
		PmArgs &p = T.p;
		p.src = p.tgt = it.pad;
		p.sWp = p.tWp = it.W + 1;
		p.smask = it.smask;
		p.tmask = it.tmask;
		p.tlist = it.tlist;
		p.sW = p.tW = it.W;
		p.sH = p.tH = it.H;
		p.nt = it.nt;
		p.shots = pm.random_shots;
		p.max_window = (pm.window != -1) ? pm.window : max(it.W, it.H);
		p.rx = a.rx;
		p.ry = a.ry;
		p.ex = a.px - a.rx;
		p.ey = a.py - a.ry;
		p.L = a.px + (grad ? 1 : 0);
		p.K = 32 / p.L;
		p.rows = a.py + (grad ? 1 : 0);
		p.lambda = a.lambda;
		p.lambda_d = a.lambda_d;
		p.seed = it.seed;
		p.calls = it.calls;
		p.smom = p.tmom = it.mom;
		p.vmax = it.mom ? it.vmax : nullptr;
		p.slopes = it.mom ? bound_slopes(dp, it.nt, ctx->num_sms) : 0;
		T.moment_tiles = moment_tiles(it.W, it.H);
		maxtiles = std::max(maxtiles, T.moment_tiles);
		p.dev = (it.mom && ctx->tune_pm_bound == 2 && dp.kind != NLI_DIST_L1_NORM) ? 1 : 0;
		p.queue = nullptr;  // the launch's queue is B.queue
		p.tile = 0;
		T.flag = it.flag;
		T.counter = it.counter;
		T.img = it.img;
		T.init = reinterpret_cast<const int2 *>(it.init);
		T.nnf_x = reinterpret_cast<int2 *>(it.out);
		const PmFields f = {T.nnf_x,   reinterpret_cast<int2 *>(it.nnf_y), it.dist_x, it.dist_y, it.hist_x, it.hist_y};
		T.io[0] = f.io(0);
		T.io[1] = f.io(1);
		maxpix = max(maxpix, it.W * it.H);
		maxpad = max(maxpad, (it.W + 1) * (it.H + 1));
		maxnt = max(maxnt, it.nt);
		total += it.nt;
		widest = (int)std::max((unsigned)widest, (unsigned)p.max_window);
	}
	cudaStream_t s = ctx->stream;
	const int per = 256;
	k_pad4_batch<<<dim3((unsigned)std::min((maxpad + per - 1) / per, 1024), (unsigned)n), per, 0, s>>>(B, C);
	NLI_CHECK_LAUNCH();
	k_fill_nnf_batch<<<dim3((unsigned)std::min((maxpix + per - 1) / per, 1024), (unsigned)n), per, 0, s>>>(B);
	NLI_CHECK_LAUNCH();
	if (B.t[0].p.smom) {
		PmFactors f;
		patch_factors(f, a);
		k_pm_moments_batch<<<dim3((unsigned)maxtiles, (unsigned)n), kMomW * kMomH, 0, s>>>(f, B);
		NLI_CHECK_LAUNCH();
		if (B.t[0].p.dev) {
			k_pm_deviations_batch<<<dim3((unsigned)std::min((maxpad + per - 1) / per, 1024), (unsigned)n), per, 0,
			                        s>>>(a, B);
			NLI_CHECK_LAUNCH();
		}
	}
	if (maxnt == 0) return;
	unsigned long long *counter = ctx->buf<unsigned long long>("pm.counter", 2);
	if (B.tile > 0) {
		const int slots = std::max(pm.iterations, 0) + 1;
		B.queue = ctx->buf<unsigned>("pm.queue", slots);
		NLI_CUDA(cudaMemsetAsync(B.queue, 0, sizeof(unsigned) * slots, s));
	}
	B.group = pm_group(total, widest, ctx->num_sms);
	long long groups = 0;
	for (int i = 0; i < n; i++) {
		B.t[i].p.group = B.group;
		groups += (B.t[i].p.nt + B.group.points - 1) / B.group.points;
	}
	const bool handled = pm_dispatch(dp.kind, C, [&](auto d) {
		d.batch(ctx, a, B, pm.iterations, groups, counter);
	});
	NLI_REQUIRE(handled, NLI_E_UNSUPPORTED, "no PatchMatch kernel for this distance / channel count");
	if (pm.iterations % 2 == 1) {
		k_copy_targets_batch<<<dim3((unsigned)std::min((maxnt + per - 1) / per, 1024), (unsigned)n), per, 0, s>>>(B);
		NLI_CHECK_LAUNCH();
	}
}

unsigned long long check_word_patchmatch()
{
	for (unsigned long long (*word)() :
	     {check_word_pm_combined, check_word_pm_combined_rgb, check_word_pm_rgbd, check_word_pm_l2, check_word_pm_l1})
		if (const unsigned long long w = word()) return w;
	return 0;
}

void patchmatch_run(nli_ctx *ctx, const nli_distance_params &dp, const nli_patchmatch_params &pm, const float *src,
                    const uint8_t *smask, int sW, int sH, const float *tgt, const uint8_t *tmask, int tW, int tH,
                    int C, const int32_t *init_nnf, int32_t *out_nnf, float *out_dist, double *energy,
                    const int32_t *tlist, int n_target, PatchMatchMetricsHost *metrics)
{
	DistArgs a;
	fill_dist_args(a, dp, C);
	NLI_REQUIRE(sW < 32768 && sH < 32768, NLI_E_UNSUPPORTED, "PatchMatch source sides must be below 32768");
	cudaStream_t s = ctx->stream;
	const int nT = tW * tH;

	// cleared before the first kernel: a memset between two would keep the second
	// from being launched early
	unsigned *vmax = ctx->tune_pm_bound ? ctx->buf<unsigned>("pm.vmax", 1) : nullptr;
	if (vmax) NLI_CUDA(cudaMemsetAsync(vmax, 0, sizeof(unsigned), s));
	// [0]: candidates evaluated, [1]: of these, at their point's match by the early-termination test
	unsigned long long *counter = ctx->buf<unsigned long long>("pm.counter", 2);
	if (energy) NLI_CUDA(cudaMemsetAsync(counter, 0, 2 * sizeof(unsigned long long), s));

	// padded float4 pixels of source and target
	float4 *s4 = ctx->buf<float4>("pm.src4", (size_t)(sW + 1) * (sH + 1));
	launch_pad4(s, src, sW, sH, C, s4);
	float4 *t4 = s4;
	if (!(tgt == src && tW == sW && tH == sH)) {
		t4 = ctx->buf<float4>("pm.tgt4", (size_t)(tW + 1) * (tH + 1));
		launch_pad4(s, tgt, tW, tH, C, t4);
	}

	if (!tlist) {
		int32_t *l = ctx->buf<int32_t>("pm.tlist", nT);
		n_target = compact_mask(ctx, tmask, tW, tH, l, "pm");
		tlist = l;
	}

	// tables of the lower bound (NLI_TUNE_PM_BOUND)
	float4 *smom = nullptr, *tmom = nullptr;
	// the deviation tables serve the L2 kinds (NLI_TUNE_PM_BOUND 2)
	const int dev = (ctx->tune_pm_bound == 2 && dp.kind != NLI_DIST_L1_NORM) ? 1 : 0;
	const int slopes = ctx->tune_pm_bound ? bound_slopes(dp, n_target, ctx->num_sms) : 0;
	if (ctx->tune_pm_bound) {
		PmFactors f;
		patch_factors(f, a);
		auto tables = [&](const char *name, const float4 *pad, int W, int H) {
			const size_t n = (size_t)(W + 1) * (H + 1);
			float4 *mom = ctx->buf<float4>(name, n * pm_moment_tables(ctx, dp, n_target));
			launch_early(s, moment_tiles(W, H), kMomW * kMomH, 0, k_pm_moments, f, pad, W, H, mom, vmax, slopes);
			NLI_CHECK_LAUNCH();
			if (dev) {
				k_pm_deviations<<<(int)((n + 255) / 256), 256, 0, s>>>(a, pad, W, H, mom);
				NLI_CHECK_LAUNCH();
			}
			return mom;
		};
		smom = tables("pm.smom", s4, sW, sH);
		tmom = t4 != s4 ? tables("pm.tmom", t4, tW, tH) : smom;
	}
	const int2 *init = reinterpret_cast<const int2 *>(init_nnf);
	if (init_nnf && init_nnf == out_nnf) {
		int2 *copy = ctx->buf<int2>("pm.init_copy", nT);
		NLI_CUDA(cudaMemcpyAsync(copy, init_nnf, sizeof(int2) * nT, cudaMemcpyDeviceToDevice, s));
		init = copy;
	}
	int2 *nnf_x = reinterpret_cast<int2 *>(out_nnf);
	int2 *nnf_y = ctx->buf<int2>("pm.nnf_y", nT);
	float *dist_x = ctx->buf<float>("pm.dist_x", nT);
	float *dist_y = ctx->buf<float>("pm.dist_y", nT);
	const PmFields b = {nnf_x,  nnf_y, dist_x, dist_y, ctx->buf<uint8_t>("pm.hist_x", nT),
	                    ctx->buf<uint8_t>("pm.hist_y", nT)};
	// the call index advances only for calls with target points, as the
	// random streams are drawn only then
	launch_early(s, (nT + 255) / 256, 256, 0, k_fill_nnf, nnf_x, out_dist, nT,
	             n_target > 0 ? &ctx->status->pm_calls : nullptr);
	NLI_CHECK_LAUNCH();
	if (n_target > 0) {
		PmArgs p;
		p.src = s4;
		p.tgt = t4;
		p.sWp = sW + 1;
		p.tWp = tW + 1;
		p.smask = smask;
		p.tmask = tmask;
		p.tlist = tlist;
		p.sW = sW;
		p.sH = sH;
		p.tW = tW;
		p.tH = tH;
		p.nt = n_target;
		p.shots = pm.random_shots;
		p.max_window = (pm.window != -1) ? pm.window : max(sW, sH);
		p.rx = a.rx;
		p.ry = a.ry;
		p.ex = a.px - a.rx;
		p.ey = a.py - a.ry;
		const bool grad = dp.kind == NLI_DIST_L2_COMBINED || dp.kind == NLI_DIST_L2_RGBD;
		p.L = a.px + (grad ? 1 : 0);
		p.K = 32 / p.L;
		p.rows = a.py + (grad ? 1 : 0);
		p.lambda = a.lambda;
		p.lambda_d = a.lambda_d;
		p.seed = ctx->seed;
		p.calls = &ctx->status->pm_calls;  // advanced by k_fill_nnf above
		p.smom = smom;
		p.tmom = tmom;
		p.vmax = vmax;
		p.slopes = slopes;
		p.dev = smom ? dev : 0;
		p.queue = nullptr;
		p.tile = ctx->tune_pm_tile;
		p.group = {32, 1};  // run_sweeps chooses
		if (p.tile > 0) {
			const int slots = std::max(pm.iterations, 0) + 1;
			p.queue = ctx->buf<unsigned>("pm.queue", slots);
			NLI_CUDA(cudaMemsetAsync(p.queue, 0, sizeof(unsigned) * slots, s));
		}
		PmMetrics mt;
		const int iters = std::max(pm.iterations, 0);
		if (metrics && iters > 0) {
			mt.energy = ctx->buf<double>("pm.m_energy", iters);
			mt.prop = ctx->buf<unsigned long long>("pm.m_prop", iters);
			mt.shots = ctx->buf<int>("pm.m_shots", 1);
			mt.partial_blocks = std::min((n_target + 255) / 256, 1024);
			mt.partials = ctx->buf<double>("pm.m_partials", mt.partial_blocks + 1);
			NLI_CUDA(cudaMemsetAsync(mt.prop, 0, sizeof(unsigned long long) * iters, s));
			NLI_CUDA(cudaMemsetAsync(mt.shots, 0, sizeof(int), s));
		}
		const bool handled = pm_dispatch(dp.kind, C, [&](auto d) {
			d.sweeps(ctx, a, p, pm.iterations, init, b, counter, mt);
		});
		NLI_REQUIRE(handled, NLI_E_UNSUPPORTED, "no PatchMatch kernel for this distance / channel count");
		const bool in_y = (pm.iterations % 2) == 1;
		const int grid = (n_target + 255) / 256;
		if (in_y || out_dist) {
			launch_early(s, grid, 256, 0, k_copy_targets, tlist, n_target, in_y ? nnf_y : nnf_x, in_y ? dist_y : dist_x,
			                                    in_y ? nnf_x : nullptr, out_dist);
			NLI_CHECK_LAUNCH();
		}
		if (energy) {
			const int eg = min(grid, 1024);
			double *partials = ctx->buf<double>("pm.energy", eg + 1);
			launch_early(s, eg, 256, 0, k_energy, tlist, n_target, in_y ? dist_y : dist_x, partials);
			NLI_CHECK_LAUNCH();
			launch_sum_partials(s, partials, eg, partials + eg);
			unsigned long long *hc = reinterpret_cast<unsigned long long *>(ctx->host_pinned);
			NLI_CUDA(cudaMemcpyAsync(hc, counter, 2 * sizeof(unsigned long long), cudaMemcpyDeviceToHost, s));
			NLI_CUDA(cudaMemcpyAsync(hc + 2, partials + eg, sizeof(double), cudaMemcpyDeviceToHost, s));
			NLI_CUDA(cudaMemcpyAsync(hc + 3, &ctx->status->timeout, sizeof(int), cudaMemcpyDeviceToHost, s));
			NLI_CUDA(cudaStreamSynchronize(s));
			if (*reinterpret_cast<const int *>(hc + 3) != 0) {
				clear_timeout(ctx);
				NLI_REQUIRE(false, NLI_E_TIMEOUT, "PatchMatch window copies timed out");
			}
			ctx->candidates += (int64_t)hc[0];
			ctx->candidates_partial += (int64_t)hc[1];
			*energy = *reinterpret_cast<double *>(hc + 2);
		}
		if (metrics && iters > 0) {
			metrics->total_distance.resize(iters);
			std::vector<unsigned long long> prop(iters);
			NLI_CUDA(cudaMemcpyAsync(metrics->total_distance.data(), mt.energy, sizeof(double) * iters,
			                         cudaMemcpyDeviceToHost, s));
			NLI_CUDA(cudaMemcpyAsync(prop.data(), mt.prop, sizeof(unsigned long long) * iters, cudaMemcpyDeviceToHost,
			                         s));
			NLI_CUDA(cudaMemcpyAsync(&metrics->max_random_shots, mt.shots, sizeof(int), cudaMemcpyDeviceToHost, s));
			NLI_CUDA(cudaStreamSynchronize(s));
			metrics->propagations.assign(prop.begin(), prop.end());
		}
	} else if (energy) {
		*energy = 0.0;
	}
}

// Device counter of evaluated candidates of the last PatchMatch calls
// (read by the multiscale driver for its statistics).
unsigned long long *pm_counter(nli_ctx *ctx) { return ctx->buf<unsigned long long>("pm.counter", 1); }

}  // namespace nli
