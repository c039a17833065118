// PatchMatch's entry points: buffers, tables and launches around the sweep
// kernels of pm_kernels.cuh, which pm_*.cu instantiate.
#include "pm_kernels.cuh"

namespace nli {

__global__ void k_pm_moments(DistArgs a, const float4 *__restrict__ pad, int W, int H, float4 *__restrict__ mom,
                             unsigned *vmax, int dev)
{
	moments_span(a, pad, W, H, mom, vmax, blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x, dev != 0);
}

// Also advances the context's PatchMatch call index when `calls` is set.
__global__ void k_fill_nnf(int2 *__restrict__ nnf, float *__restrict__ dist, int n, unsigned long long *calls)
{
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
	const int i = blockIdx.x * blockDim.x + threadIdx.x;
	if (i >= nt) return;
	const int pix = tlist[i];
	if (nnf_dst) nnf_dst[pix] = nnf_src[pix];
	if (dist_dst) dist_dst[pix] = dist_src[pix];
}

__global__ void k_energy(const int32_t *__restrict__ tlist, int nt, const float *__restrict__ dist,
                         double *__restrict__ partials)
{
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
	k_energy<<<m.partial_blocks, 256, 0, s>>>(p.tlist, p.nt, dist, m.partials);
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

// The patch means of every active image (k_pm_moments per image).
__global__ void k_pm_moments_batch(DistArgs a, const __grid_constant__ PmBatchArgs B)
{
	const int t = blockIdx.y;
	const PmBatchTask &T = B.t[t];
	if (!batch_on(B.active, T.flag) || !T.p.smom) return;
	moments_span(a, T.p.src, T.p.sW, T.p.sH, const_cast<float4 *>(T.p.smom), const_cast<unsigned *>(T.p.vmax),
	             blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x, T.p.dev != 0);
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
		// the item's table holds room for the deviations (4 tables)
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
		k_pm_moments_batch<<<dim3((unsigned)std::min((maxpad + per - 1) / per, 1024), (unsigned)n), per, 0, s>>>(a,
		                                                                                                       B);
		NLI_CHECK_LAUNCH();
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

	// padded float4 pixels of source and target
	float4 *s4 = ctx->buf<float4>("pm.src4", (size_t)(sW + 1) * (sH + 1));
	launch_pad4(s, src, sW, sH, C, s4);
	float4 *t4 = s4;
	if (!(tgt == src && tW == sW && tH == sH)) {
		t4 = ctx->buf<float4>("pm.tgt4", (size_t)(tW + 1) * (tH + 1));
		launch_pad4(s, tgt, tW, tH, C, t4);
	}

	// patch means for the lower bound (NLI_TUNE_PM_BOUND)
	float4 *smom = nullptr, *tmom = nullptr;
	unsigned *vmax = nullptr;
	// the deviation tables serve the L2 kinds (NLI_TUNE_PM_BOUND 2)
	const int dev = (ctx->tune_pm_bound == 2 && dp.kind != NLI_DIST_L1_NORM) ? 1 : 0;
	if (ctx->tune_pm_bound) {
		DistArgs da;
		fill_dist_args(da, dp, C);
		vmax = ctx->buf<unsigned>("pm.vmax", 1);
		NLI_CUDA(cudaMemsetAsync(vmax, 0, sizeof(unsigned), s));
		const int ns = (sW + 1) * (sH + 1);
		smom = ctx->buf<float4>("pm.smom", (size_t)ns * (dev ? 4 : 1));
		k_pm_moments<<<(ns + 255) / 256, 256, 0, s>>>(da, s4, sW, sH, smom, vmax, dev);
		NLI_CHECK_LAUNCH();
		tmom = smom;
		if (t4 != s4) {
			const int nt4 = (tW + 1) * (tH + 1);
			tmom = ctx->buf<float4>("pm.tmom", (size_t)nt4 * (dev ? 4 : 1));
			k_pm_moments<<<(nt4 + 255) / 256, 256, 0, s>>>(da, t4, tW, tH, tmom, vmax, dev);
			NLI_CHECK_LAUNCH();
		}
	}

	if (!tlist) {
		int32_t *l = ctx->buf<int32_t>("pm.tlist", nT);
		n_target = compact_mask(ctx, tmask, tW, tH, l, "pm");
		tlist = l;
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
	// [0]: candidates evaluated, [1]: of these, stopped after the first 32 taps
	unsigned long long *counter = ctx->buf<unsigned long long>("pm.counter", 2);
	// the call index advances only for calls with target points, as the
	// random streams are drawn only then
	k_fill_nnf<<<(nT + 255) / 256, 256, 0, s>>>(nnf_x, out_dist, nT, n_target > 0 ? &ctx->status->pm_calls : nullptr);
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
		p.dev = smom ? dev : 0;
		p.queue = nullptr;
		p.tile = ctx->tune_pm_tile;
		p.group = {32, 1};  // run_sweeps chooses
		if (p.tile > 0) {
			const int slots = std::max(pm.iterations, 0) + 1;
			p.queue = ctx->buf<unsigned>("pm.queue", slots);
			NLI_CUDA(cudaMemsetAsync(p.queue, 0, sizeof(unsigned) * slots, s));
		}
		if (energy) NLI_CUDA(cudaMemsetAsync(counter, 0, 2 * sizeof(unsigned long long), s));
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
			k_copy_targets<<<grid, 256, 0, s>>>(tlist, n_target, in_y ? nnf_y : nnf_x, in_y ? dist_y : dist_x,
			                                    in_y ? nnf_x : nullptr, out_dist);
			NLI_CHECK_LAUNCH();
		}
		if (energy) {
			const int eg = min(grid, 1024);
			double *partials = ctx->buf<double>("pm.energy", eg + 1);
			k_energy<<<eg, 256, 0, s>>>(tlist, n_target, in_y ? dist_y : dist_x, partials);
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
