// AImageUpdating subclasses as gather kernels over the nearest-neighbour
// field:
//   NL-means   (patch_non_local_means.cpp:23-100)   - one thread per hole pixel
//              and channel
//   NL-medians (patch_non_local_medians.cpp:23-127) - one warp per hole pixel
//   NL-Poisson (patch_non_local_poisson.cpp:36-477) - coefficient gather,
//              right-hand side, and the conjugate gradient of every channel
//              in one launch: a CTA, a cluster or all SMs, by the system's size
//   NL-depth   (patch_non_local_depth.cpp:36-55)    - NL-Poisson with a
//              per-channel lambda on the 4-channel image, orig = image
#include <cooperative_groups.h>

#include <atomic>
#include <cmath>
#include <type_traits>

#include "nli_device.cuh"

namespace nli {

struct UpdArgs {
	int px, py, hx, hy;
	int W, H, C;
	float weights[kMaxTaps];
};

static void fill_upd_args(UpdArgs &u, const nli_update_params &p, int W, int H, int C)
{
	NLI_REQUIRE(p.patch_x >= 1 && p.patch_y >= 1 && p.patch_x <= NLI_MAX_PATCH && p.patch_y <= NLI_MAX_PATCH,
	            NLI_E_UNSUPPORTED, "patch size outside 1.." + std::to_string(NLI_MAX_PATCH));
	std::memset(&u, 0, sizeof(u));
	u.px = p.patch_x;
	u.py = p.patch_y;
	u.hx = p.patch_x / 2;
	u.hy = p.patch_y / 2;
	u.W = W;
	u.H = H;
	u.C = C;
	std::vector<float> w = gaussian_weights_host(p.patch_x, p.patch_y, p.sigma, p.sigma);
	std::memcpy(u.weights, w.data(), sizeof(float) * w.size());
}

// ------------------------------------------------------------- NL-means
// Reference arithmetic: float accumulators, separate roundings, the patch
// weight indexed from the clipped window corner (:71), confidence applied
// inside the domain only (:72-74).  New values go to a compact buffer and
// are scattered afterwards, so every pixel reads the pre-update image.
//
// One thread per hole pixel and channel.  The sums are sequential by the
// reference's order, so what a pixel takes is its chain of dependent loads
// (field, then the pixel it names): a column of the window is loaded at a
// time, nine of each in flight.  With one thread per pixel and one tap at a
// time a 256 x 256 level (3300 hole pixels) took 56 us, and the 256 x 256 NL-means
// process() 49.0 ms; now 43.3 ms.
constexpr int kMeansGroup = 9;  // rows of a window column loaded together

// The new value of channel c at hole pixel pix; its square difference is
// returned.  u supplies the patch and its weights; W, H, C are the image's.
__device__ __forceinline__ float nlmeans_value(const UpdArgs &u, int W, int H, int C, int c,
                                               const float *__restrict__ img, int pix, const uint8_t *__restrict__ dom,
                                               const int2 *__restrict__ nnf, const float *__restrict__ conf, float &out)
{
	if (!nli_in_bounds(pix, (long long)W * H, kSiteHole)) return 0.f;
	const int x = pix % W, y = pix / W;
	const int x_a = max(x - u.hx, 0), x_b = min(x + u.hx, W - 1);
	const int y_a = max(y - u.hy, 0), y_b = min(y + u.hy, H - 1);
	float tv = 0.f, tw = 0.f;
	for (int ii = x_a; ii <= x_b; ii++)
		for (int j0 = y_a; j0 <= y_b; j0 += kMeansGroup) {
			int2 q[kMeansGroup];
			float cf[kMeansGroup], s[kMeansGroup];
			bool ok[kMeansGroup], damped[kMeansGroup];
#pragma unroll
			for (int g = 0; g < kMeansGroup; g++) {
				const int at = min(j0 + g, y_b) * W + ii;
				q[g] = nnf[at];
				damped[g] = conf && dom[at];
				cf[g] = conf ? conf[at] : 0.f;
			}
#pragma unroll
			for (int g = 0; g < kMeansGroup; g++) {
				const int jj = j0 + g;
				ok[g] = jj <= y_b && q[g].x != -1;
				q[g].x += x - ii;
				q[g].y += y - jj;
				ok[g] = ok[g] && q[g].x >= 0 && q[g].y >= 0 && q[g].x < W && q[g].y < H &&
				        nli_in_bounds((long long)q[g].y * W + q[g].x, (long long)W * H, kSiteMeansSource);
				s[g] = img[(size_t)C * (ok[g] ? q[g].y * W + q[g].x : pix) + c];
			}
#pragma unroll
			for (int g = 0; g < kMeansGroup; g++) {
				if (!ok[g]) continue;
				float w = u.weights[(j0 + g - y_a) * u.px + (ii - x_a)];
				if (damped[g]) w = fm(w, cf[g]);
				tw = fa(tw, w);
				tv = fa(tv, fm(s[g], w));
			}
		}
	const float prev = img[(size_t)C * pix + c];
	out = prev;
	if (!(tw > 0.0f)) return 0.f;
	out = __fdiv_rn(tv, tw);
	const float d = fs(prev, out);
	return fm(d, d);
}

__global__ void __launch_bounds__(256) k_nlmeans(UpdArgs u, const float *__restrict__ img,
                                                 const int32_t *__restrict__ hole, int nh,
                                                 const uint8_t *__restrict__ dom, const int2 *__restrict__ nnf,
                                                 const float *__restrict__ conf, float *__restrict__ newval,
                                                 double *__restrict__ partials)
{
	next_launch_may_start();
	previous_launch_done();
	__shared__ double red[8];
	const int i = blockIdx.x * blockDim.x + threadIdx.x;
	const int k = i / u.C, c = i - k * u.C;
	float sq = 0.f;
	if (k < nh) sq = nlmeans_value(u, u.W, u.H, u.C, c, img, hole[k], dom, nnf, conf, newval[i]);
	const double acc = block_sum<256>((double)sq, red);
	if (threadIdx.x == 0) partials[blockIdx.x] = acc;
}

__global__ void k_scatter_values(const int32_t *__restrict__ hole, int nh, int C, const float *__restrict__ newval,
                                 float *__restrict__ img)
{
	next_launch_may_start();
	previous_launch_done();
	const int i = blockIdx.x * blockDim.x + threadIdx.x;
	if (i >= nh * C) return;
	const int k = i / C, c = i % C;
	img[(size_t)C * hole[k] + c] = newval[i];
}

// ------------------------------------------------------------ NL-medians
// One warp per hole pixel.  The candidates of the window are numbered in the
// reference's order (x outer, y inner, :61-62) and held 32 to a block, one per
// lane; per channel each is ranked by value against all others (ties by
// number), scattered to its place in sorted order, and the weighted median is
// found by the reference's sequential subtraction (:110-127), one channel per
// lane.
//
// Bound by issue: 81 x 81 comparisons a channel.  A candidate of an earlier
// block counts when it is not greater, one of the same or a later block when
// it is less, and equals within a block are told apart by one match, so a
// comparison is two instructions on registers and a quarter of a load (six
// and a whole one when every pair tested value and number).  382 x 388 with
// 22 000 hole pixels: 159 us so, 89 us now.
constexpr int kMedWarps = 4;

// Blocks of 32 candidates the kernels are compiled for: up to 9 x 9 patches,
// and the largest.
constexpr int kMedSmall = 3, kMedLarge = (kMaxTaps + 31) / 32;

// Shared memory of one NL-medians warp.
template <int NB>
struct MedSmem {
	float val[4][32 * NB];  // per channel: the candidates' values, then sorted
	float sw[4][32 * NB];   // the sorted ones' weights
	float w[32 * NB];
};

// Moves one channel's m values (in B blocks of 32) and their weights to their
// places in sorted order.
template <int B>
__device__ __forceinline__ void med_sort(float *val, float *sw, const float *w, int m)
{
	const int lane = threadIdx.x & 31;
	float v[B];
	int rank[B];
#pragma unroll
	for (int b = 0; b < B; b++) {
		v[b] = val[32 * b + lane];
		// equals of lower numbers in the block (+0 and -0 are equal)
		rank[b] = __popc(__match_any_sync(0xffffffffu, __float_as_uint(v[b] + 0.0f)) & ((1u << lane) - 1u));
	}
#pragma unroll
	for (int jb = 0; jb < B; jb++)
#pragma unroll 2  // more would hold every load's registers and leave fewer warps
		for (int j = 0; j < 32; j += 4) {
			const float4 o4 = *reinterpret_cast<const float4 *>(val + 32 * jb + j);
			const float o[4] = {o4.x, o4.y, o4.z, o4.w};
#pragma unroll
			for (int i = 0; i < 4; i++)
#pragma unroll
				for (int b = 0; b < B; b++) rank[b] += (jb < b ? o[i] <= v[b] : o[i] < v[b]) ? 1 : 0;
		}
	__syncwarp();
#pragma unroll
	for (int b = 0; b < B; b++)
		if (32 * b + lane < m) {
			val[rank[b]] = v[b];
			sw[rank[b]] = w[32 * b + lane];
		}
}

// med_sort for the number of blocks that m values take (NB at most).
template <int NB>
__device__ __forceinline__ void med_rank_blocks(float *val, float *sw, const float *w, int m)
{
	if constexpr (NB > 1)
		if (m <= 32 * (NB - 1)) return med_rank_blocks<NB - 1>(val, sw, w, m);
	med_sort<NB>(val, sw, w, m);
}

// One hole pixel, computed by one whole warp: lanes 0..C-1 write the new
// values into out[0..C), lane 0 returns (u_old - u_new)^2 summed over the
// channels.
template <int NB>
__device__ __forceinline__ double nlmedians_pixel(const UpdArgs &u, int W, int H, int C,
                                                  const float *__restrict__ img, int pix,
                                                  const uint8_t *__restrict__ dom, const int2 *__restrict__ nnf,
                                                  const float *__restrict__ conf, float *__restrict__ out,
                                                  MedSmem<NB> &sm)
{
	const int lane = threadIdx.x & 31;
	if (!nli_in_bounds(pix, (long long)W * H, kSiteHole)) return 0.0;
	const int x = pix % W, y = pix / W;
	const int x_a = max(x - u.hx, 0), x_b = min(x + u.hx, W - 1);
	const int y_a = max(y - u.hy, 0), y_b = min(y + u.hy, H - 1);
	const int ny = y_b - y_a + 1;
	const int total = (x_b - x_a + 1) * ny;
	// collect valid candidates in reference order (compacted)
	int m = 0;
	for (int base = 0; base < total; base += 32) {
		const int k = base + lane;
		bool valid = false;
		float w = 0.f;
		int qx = 0, qy = 0;
		if (k < total) {
			const int ii = x_a + k / ny, jj = y_a + k % ny;
			int2 q = nnf[jj * W + ii];
			if (q.x != -1) {
				qx = q.x + x - ii;
				qy = q.y + y - jj;
				if (qx >= 0 && qy >= 0 && qx < W && qy < H &&
				    nli_in_bounds((long long)qy * W + qx, (long long)W * H, kSiteMeansSource)) {
					valid = true;
					w = u.weights[(jj - y_a) * u.px + (ii - x_a)];
					if (conf && dom[jj * W + ii]) w = fm(w, conf[jj * W + ii]);
				}
			}
		}
		const unsigned bal = __ballot_sync(0xffffffffu, valid);
		if (valid) {
			const int slot = m + __popc(bal & ((1u << lane) - 1u));
			sm.w[slot] = w;
			for (int c = 0; c < C; c++) sm.val[c][slot] = img[(size_t)C * (qy * W + qx) + c];
		}
		m += __popc(bal);
	}
	if (m == 0) {
		if (lane < C) out[lane] = img[(size_t)C * pix + lane];
		return 0.0;
	}
	// the last block's free places: behind every value, and of no weight
	for (int k = m + lane; k < ((m + 31) & ~31); k += 32) {
		sm.w[k] = 0.f;
		for (int c = 0; c < C; c++) {
			sm.val[c][k] = __int_as_float(0x7f800000);
			sm.sw[c][k] = 0.f;
		}
	}
	__syncwarp();
	for (int c = 0; c < C; c++) med_rank_blocks<NB>(sm.val[c], sm.sw[c], sm.w, m);
	__syncwarp();
	float sq = 0.f;
	if (lane < C) {
		// total weight, summed in candidate order (:80); four weights to a
		// load, those past the last being 0
		float tw = 0.f;
		for (int k = 0; k < m; k += 4) {
			const float4 w = *reinterpret_cast<const float4 *>(&sm.w[k]);
			tw = fa(fa(fa(fa(tw, w.x), w.y), w.z), w.w);
		}
		float median = 0.0f, t = tw;
		const float half = tw / 2;
		for (int k = 0; k < m; k += 4) {
			const float4 w = *reinterpret_cast<const float4 *>(&sm.sw[lane][k]);
			const float t0 = fs(t, w.x), t1 = fs(t0, w.y), t2 = fs(t1, w.z);
			t = fs(t2, w.w);
			if (t0 < half || t1 < half || t2 < half || t < half) {
				median = sm.val[lane][k + (t0 < half ? 0 : t1 < half ? 1 : t2 < half ? 2 : 3)];
				break;
			}
		}
		const float d = fs(img[(size_t)C * pix + lane], median);
		sq = fm(d, d);
		out[lane] = median;
	}
	double acc = 0.0;
	for (int c = 0; c < C; c++) acc += (double)__shfl_sync(0xffffffffu, sq, c);
	__syncwarp();
	return acc;
}

// Candidates of a window at most (even sides reach one further).
static int med_window(const UpdArgs &u) { return (2 * u.hx + 1) * (2 * u.hy + 1); }

template <int NB>
__global__ void __launch_bounds__(32 * kMedWarps) k_nlmedians(UpdArgs u, const float *__restrict__ img,
                                                              const int32_t *__restrict__ hole, int nh,
                                                              const uint8_t *__restrict__ dom,
                                                              const int2 *__restrict__ nnf,
                                                              const float *__restrict__ conf,
                                                              float *__restrict__ newval, double *__restrict__ partials)
{
	next_launch_may_start();
	previous_launch_done();
	__shared__ __align__(16) MedSmem<NB> sm[kMedWarps];
	__shared__ double red[kMedWarps];
	const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
	const int i = blockIdx.x * kMedWarps + wid;
	double acc = 0.0;
	if (i < nh)
		acc = nlmedians_pixel<NB>(u, u.W, u.H, u.C, img, hole[i], dom, nnf, conf, newval + (size_t)u.C * i, sm[wid]);
	if (lane == 0) red[wid] = acc;
	__syncthreads();
	if (threadIdx.x == 0) {
		double t = 0.0;
		for (int w = 0; w < kMedWarps; w++) t += red[w];
		partials[blockIdx.x] = t;
	}
}

// ------------------------------------------------------------ NL-Poisson
// Coefficients of calculate_pde_coefficients (:139-232) as a gather: pixel
// q receives, from every extended-domain centre c whose window holds q
// (visited in raster order), w = conf(c) * g(q - c) and the image / gradient
// at n = nnf(c) + q - c when n lies in the image.  Stored unscaled:
//   S = sum w, U_c = sum w u_c(n), GX_c = sum w gx_c(n), GY_c = sum w gy_c(n);
// a1 = lambda S, a2 = (1-lambda) S, f1 = lambda U, F = (1-lambda) G.
// The pixels computed are the hole pixels and their left / upper
// neighbours (all that the right-hand side and the stencil read).
struct CoefOut {
	float *S;   // W*H
	float *U;   // W*H*C
	float *GX;  // W*H*C
	float *GY;  // W*H*C
};

// The image is read as padded float4 pixels (launch_pad4): a pixel and its
// forward differences are three of them, differences across the last column
// and row being 0 (gradient.cpp:37-63).
struct Pix3 {
	float4 v, gx, gy;
};

__device__ __forceinline__ Pix3 load_pix3(const float4 *__restrict__ pad, int W, int H, int x, int y)
{
	const float4 *p = pad + (size_t)y * (W + 1) + x;
	const float4 v = __ldg(p), r = __ldg(p + 1), d = __ldg(p + W + 1);
	const bool mx = x != W - 1, my = y != H - 1;
	Pix3 t;
	t.v = v;
	t.gx = make_float4(mx ? fs(r.x, v.x) : 0.f, mx ? fs(r.y, v.y) : 0.f, mx ? fs(r.z, v.z) : 0.f, mx ? fs(r.w, v.w) : 0.f);
	t.gy = make_float4(my ? fs(d.x, v.x) : 0.f, my ? fs(d.y, v.y) : 0.f, my ? fs(d.z, v.z) : 0.f, my ? fs(d.w, v.w) : 0.f);
	return t;
}

// a + w v over the first C components
template <int C>
__device__ __forceinline__ void add_wc(float4 &a, float w, const float4 &v)
{
	a.x = fmaf(w, v.x, a.x);
	if (C > 1) a.y = fmaf(w, v.y, a.y);
	if (C > 2) a.z = fmaf(w, v.z, a.z);
	if (C > 3) a.w = fmaf(w, v.w, a.w);
}

template <int C>
__device__ __forceinline__ void store_c(float *p, const float4 &v)
{
	p[0] = v.x;
	if (C > 1) p[1] = v.y;
	if (C > 2) p[2] = v.z;
	if (C > 3) p[3] = v.w;
}

// The sums of one coefficient pixel.
struct CoefSum {
	float S;
	float4 U, GX, GY;
};

template <int C>
__device__ __forceinline__ void store_coef(const CoefOut &out, int q, const CoefSum &a)
{
	out.S[q] = a.S;
	store_c<C>(out.U + (size_t)C * q, a.U);
	store_c<C>(out.GX + (size_t)C * q, a.GX);
	store_c<C>(out.GY + (size_t)C * q, a.GY);
}

template <int C>
__device__ __forceinline__ void gather_coef(const UpdArgs &u, int W, int H, int qx, int qy,
                                            const uint8_t *__restrict__ ext, const int2 *__restrict__ nnf,
                                            const float *__restrict__ conf, const float4 *__restrict__ pad, CoefOut out)
{
	const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
	CoefSum a = {0.f, zero, zero, zero};
	const int cy0 = max(qy - u.hy, 0), cy1 = min(qy + u.hy, H - 1);
	const int cx0 = max(qx - u.hx, 0), cx1 = min(qx + u.hx, W - 1);
	for (int cy = cy0; cy <= cy1; cy++)
		for (int cx = cx0; cx <= cx1; cx++) {
			const int c = cy * W + cx;
			if (!ext[c]) continue;
			const int2 nb = nnf[c];
			const int nx = nb.x + qx - cx, ny = nb.y + qy - cy;
			if (nx < 0 || ny < 0 || nx >= W || ny >= H) continue;
			float w = u.weights[(qy - cy + u.hy) * u.px + (qx - cx + u.hx)];
			if (conf) w = conf[c] * w;
			const Pix3 t = load_pix3(pad, W, H, nx, ny);
			a.S += w;
			add_wc<C>(a.U, w, t.v);
			add_wc<C>(a.GX, w, t.gx);
			add_wc<C>(a.GY, w, t.gy);
		}
	store_coef<C>(out, qy * W + qx, a);
}

// Hole pixel k and the neighbours it owns (see k_poisson_coef).
template <int C>
__device__ __forceinline__ void coef_hole_pixel(const UpdArgs &u, int W, int H, int k, const int32_t *__restrict__ hole,
                                                const uint8_t *__restrict__ dom, const uint8_t *__restrict__ ext,
                                                const int2 *__restrict__ nnf, const float *__restrict__ conf,
                                                const float4 *__restrict__ pad, CoefOut out, int32_t *__restrict__ index)
{
	const int pix = hole[k];
	const int x = pix % W, y = pix / W;
	index[pix] = k;
	gather_coef<C>(u, W, H, x, y, ext, nnf, conf, pad, out);
	// left neighbour: owned by this hole pixel when it is not a hole pixel
	if (x > 0 && !dom[pix - 1]) gather_coef<C>(u, W, H, x - 1, y, ext, nnf, conf, pad, out);
	// upper neighbour: owned here when it is neither a hole pixel nor the left
	// neighbour of a hole pixel (then its right neighbour owns it)
	if (y > 0 && !dom[pix - W] && !(x + 1 < W && dom[pix - W + 1]))
		gather_coef<C>(u, W, H, x, y - 1, ext, nnf, conf, pad, out);
}

template <int C>
__global__ void __launch_bounds__(128) k_poisson_coef(UpdArgs u, const int32_t *__restrict__ hole, int nh,
                                                      const uint8_t *__restrict__ dom,
                                                      const uint8_t *__restrict__ ext, const int2 *__restrict__ nnf,
                                                      const float *__restrict__ conf, const float4 *__restrict__ pad,
                                                      CoefOut out, int32_t *__restrict__ index)
{
	next_launch_may_start();
	previous_launch_done();
	const int i = blockIdx.x * blockDim.x + threadIdx.x;
	if (i >= nh) return;
	coef_hole_pixel<C>(u, u.W, u.H, i, hole, dom, ext, nnf, conf, pad, out, index);
}

// Item `item` of 3 nh (thread group of 8 lanes, `sub` = lane within the
// group): the coefficients of hole pixel `item` for the first nh, then of the
// left and upper neighbours of the hole pixels where these are owned.  Also
// writes the hole pixels' unknown index.
template <int C>
__device__ __forceinline__ void coef8_item(const UpdArgs &u, int W, int H, int item, int sub,
                                           const int32_t *__restrict__ hole, int nh, const uint8_t *__restrict__ dom,
                                           const uint8_t *__restrict__ ext, const int2 *__restrict__ nnf,
                                           const float *__restrict__ conf, const float4 *__restrict__ pad, CoefOut out,
                                           int32_t *__restrict__ index)
{
	if (item >= 3 * nh) return;
	const int k = item < nh ? item : (item - nh) >> 1;
	const int pix = hole[k];
	if (!nli_in_bounds(pix, (long long)W * H, kSiteHole)) return;  // the item's 8 lanes leave together
	int qx = pix % W, qy = pix / W;
	bool owned = true;
	if (item < nh) {
		if (sub == 0) index[pix] = k;
	} else if (((item - nh) & 1) == 0) {
		owned = qx > 0 && !dom[pix - 1];
		qx--;
	} else {
		owned = qy > 0 && !dom[pix - W] && !(qx + 1 < W && dom[pix - W + 1]);
		qy--;
	}
	// all 8 lanes of an item agree on `owned`; whole groups leave together
	if (!owned) return;
	const unsigned gmask = 0xffu << (threadIdx.x & 24);
	const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
	CoefSum a = {0.f, zero, zero, zero};
	const int taps = u.px * u.py;
	// a lane's taps in groups whose loads are in flight together; a tap
	// without a centre reads the pixel itself and adds nothing
	constexpr int kGroup = 4;
	for (int t0 = sub; t0 < taps; t0 += 8 * kGroup) {
		int2 nb[kGroup];
		float w[kGroup];
		bool ok[kGroup];
		int dx[kGroup], dy[kGroup];
#pragma unroll
		for (int i = 0; i < kGroup; i++) {
			const int t = t0 + 8 * i;
			const int ty = t / u.px, tx = t - ty * u.px;
			// centre c = q - (tap offset), tap offset = (tx - hx, ty - hy)
			dx[i] = tx - u.hx;
			dy[i] = ty - u.hy;
			const int cx = qx - dx[i], cy = qy - dy[i];
			ok[i] = t < taps && cx >= 0 && cy >= 0 && cx < W && cy < H;
			const int c = ok[i] ? cy * W + cx : pix;
			ok[i] = ok[i] && ext[c];
			nb[i] = nnf[c];
			w[i] = t < taps ? u.weights[t] : 0.f;
			if (conf) w[i] = conf[c] * w[i];
		}
		Pix3 v[kGroup];
#pragma unroll
		for (int i = 0; i < kGroup; i++) {
			const int nx = nb[i].x + dx[i], ny = nb[i].y + dy[i];
			ok[i] = ok[i] && nx >= 0 && ny >= 0 && nx < W && ny < H &&
			        nli_in_bounds((long long)ny * W + nx, (long long)W * H, kSiteCoefSource);
			v[i] = load_pix3(pad, W, H, ok[i] ? nx : qx, ok[i] ? ny : qy);
		}
#pragma unroll
		for (int i = 0; i < kGroup; i++) {
			if (!ok[i]) continue;
			a.S += w[i];
			add_wc<C>(a.U, w[i], v[i].v);
			add_wc<C>(a.GX, w[i], v[i].gx);
			add_wc<C>(a.GY, w[i], v[i].gy);
		}
	}
	auto fold = [gmask](float4 &v, int o) {
		v.x += __shfl_xor_sync(gmask, v.x, o);
		if (C > 1) v.y += __shfl_xor_sync(gmask, v.y, o);
		if (C > 2) v.z += __shfl_xor_sync(gmask, v.z, o);
		if (C > 3) v.w += __shfl_xor_sync(gmask, v.w, o);
	};
#pragma unroll
	for (int o = 4; o > 0; o >>= 1) {
		a.S += __shfl_xor_sync(gmask, a.S, o);
		fold(a.U, o);
		fold(a.GX, o);
		fold(a.GY, o);
	}
	if (sub == 0) store_coef<C>(out, qy * W + qx, a);
}

// The same gather with 8 lanes per coefficient pixel: lane j of an item's 8
// takes window taps j, j + 8, ...; the 8 partial sums are added with
// shuffles.  Same terms as gather_coef, summed in a tree.  Bound by L1 and the
// latency of the gathers.  The hole pixels come first, so that whole warps of
// neighbour items that are not owned (nearly all) leave at once: interleaved
// with them, two thirds of every warp's lanes were idle, and with ten scalar
// loads per tap (pixel and gradient image) instead of three float4 a 512 x 512
// hole of 39 000 pixels took 92.5 us; this takes 38.8 (1024 x 685, 175 000
// pixels: 366 and 139 us).
template <int C>
__global__ void __launch_bounds__(256) k_poisson_coef8(UpdArgs u, const int32_t *__restrict__ hole, int nh,
                                                       const uint8_t *__restrict__ dom,
                                                       const uint8_t *__restrict__ ext, const int2 *__restrict__ nnf,
                                                       const float *__restrict__ conf, const float4 *__restrict__ pad,
                                                       CoefOut out, int32_t *__restrict__ index)
{
	next_launch_may_start();
	previous_launch_done();
	coef8_item<C>(u, u.W, u.H, (blockIdx.x * blockDim.x + threadIdx.x) >> 3, threadIdx.x & 7, hole, nh, dom, ext, nnf,
	              conf, pad, out, index);
}

// Calls f with the channel count as a compile-time constant.
template <class F>
static void with_channels(int C, F &&f)
{
	if (C == 1) f(std::integral_constant<int, 1>());
	if (C == 2) f(std::integral_constant<int, 2>());
	if (C == 3) f(std::integral_constant<int, 3>());
	if (C == 4) f(std::integral_constant<int, 4>());
}

// Per unknown (hole pixel) data of the symmetric system
//   (a1 - div a2 grad) delta = b,  delta = 0 outside the hole,
// with the anisotropic Laplacian of calculate_anisotropic_laplacian
// (:291-356): links up/left take a2 of the neighbour, down/right take a2
// of the centre, links that leave the image are absent.
struct Unknown {
	float S;         // unscaled a1 / a2 at the centre
	float s_up, s_left, s_down, s_right;  // unscaled link coefficients (0 if no link)
	int n_up, n_left, n_down, n_right;    // unknown index of the neighbour, -1 if not a hole pixel
};

struct PoissonArgs {
	int W, H, C, nh;
	float lambda[4];
	float tol;
	int limit;
};

// The cluster CG's record: neighbours as 16-bit codes (owning CTA << 12 | index
// within its range, kNoNb for none).
constexpr int kNoNb = 0xFFFF;

struct UnkC {
	float S, s_up, s_left;
	uint32_t ud;     // up code << 16 | down code
	uint32_t lr;     // left code << 16 | right code
	uint32_t links;  // bit 0: down link inside the image, bit 1: right link inside the image
};

// Right-hand side b and initial perturbation delta0 = image - orig
// (patch_non_local_poisson.cpp:62-82), and the per-unknown system data: the
// cluster CG's record for ranges of `chunk` unknowns, or (chunk 0) the grid
// CG's.  hole_index holds the unknown index of the hole pixels only.
__device__ __forceinline__ void poisson_setup_unknown(const PoissonArgs &a, int chunk, int k,
                                                      const int32_t *__restrict__ hole,
                                                      const uint8_t *__restrict__ dom,
                                                      const int32_t *__restrict__ hole_index, CoefOut co,
                                                      const float *__restrict__ img, const float *__restrict__ orig,
                                                      Unknown *__restrict__ unk, UnkC *__restrict__ unkc,
                                                      float *__restrict__ b, float *__restrict__ x0)
{
	const int W = a.W, H = a.H, C = a.C;
	const int pix = hole[k];
	const int x = pix % W, y = pix / W;
	Unknown n;
	n.S = co.S[pix];
	n.s_up = (y != 0) ? co.S[pix - W] : 0.f;
	n.s_left = (x != 0) ? co.S[pix - 1] : 0.f;
	n.s_down = (y != H - 1) ? n.S : 0.f;
	n.s_right = (x != W - 1) ? n.S : 0.f;
	auto at = [&](bool inside, int p) { return inside && dom[p] ? hole_index[p] : -1; };
	n.n_up = at(y != 0, pix - W);
	n.n_left = at(x != 0, pix - 1);
	n.n_down = at(y != H - 1, pix + W);
	n.n_right = at(x != W - 1, pix + 1);
	if (chunk > 0) {
		auto code = [chunk](int m) -> uint32_t {
			return (m >= 0) ? (uint32_t)(((m / chunk) << 12) | (m % chunk)) : (uint32_t)kNoNb;
		};
		UnkC c;
		c.S = n.S;
		c.s_up = n.s_up;
		c.s_left = n.s_left;
		c.ud = (code(n.n_up) << 16) | code(n.n_down);
		c.lr = (code(n.n_left) << 16) | code(n.n_right);
		c.links = ((y != H - 1) ? 1u : 0u) | ((x != W - 1) ? 2u : 0u);
		unkc[k] = c;
	} else {
		unk[k] = n;
	}
	for (int c = 0; c < C; c++) {
		const float lam = a.lambda[c], oml = 1.0f - lam;
		const float a1 = lam * n.S;
		const float f1 = lam * co.U[(size_t)C * pix + c];
		// backward divergence of F = (1-lambda) G on the domain (:235-285)
		float f2 = 0.f;
		if (lam != 1.0f) {
			const float fx = oml * co.GX[(size_t)C * pix + c];
			const float fy = oml * co.GY[(size_t)C * pix + c];
			const float fxl = (x > 0) ? oml * co.GX[(size_t)C * (pix - 1) + c] : 0.f;
			const float fyu = (y > 0) ? oml * co.GY[(size_t)C * (pix - W) + c] : 0.f;
			f2 = (x == 0) ? fx : (x == W - 1) ? -fxl : fx - fxl;
			f2 += (y == 0) ? fy : (y == H - 1) ? -fyu : fy - fyu;
		}
		// anisotropic Laplacian of the original image at the hole pixel
		const float o = orig[(size_t)C * pix + c];
		const float ou = (y != 0) ? orig[(size_t)C * (pix - W) + c] : 0.f;
		const float ol = (x != 0) ? orig[(size_t)C * (pix - 1) + c] : 0.f;
		const float od = (y != H - 1) ? orig[(size_t)C * (pix + W) + c] : 0.f;
		const float orr = (x != W - 1) ? orig[(size_t)C * (pix + 1) + c] : 0.f;
		const float lap = oml * (n.s_up * ou + n.s_left * ol + n.s_down * od + n.s_right * orr -
		                         o * (n.s_up + n.s_left + n.s_down + n.s_right));
		b[(size_t)c * a.nh + k] = f1 - f2 - a1 * o + lap;
		x0[(size_t)c * a.nh + k] = img[(size_t)C * pix + c] - o;
	}
}

__global__ void k_poisson_setup(PoissonArgs a, int chunk, const int32_t *__restrict__ hole,
                                const uint8_t *__restrict__ dom, const int32_t *__restrict__ hole_index, CoefOut co,
                                const float *__restrict__ img, const float *__restrict__ orig,
                                Unknown *__restrict__ unk, UnkC *__restrict__ unkc, float *__restrict__ b,
                                float *__restrict__ x0)
{
	next_launch_may_start();
	previous_launch_done();
	const int k = blockIdx.x * blockDim.x + threadIdx.x;
	if (k >= a.nh) return;
	poisson_setup_unknown(a, chunk, k, hole, dom, hole_index, co, img, orig, unk, unkc, b, x0);
}

__device__ __forceinline__ float apply_A(const Unknown &n, float lam, const float *__restrict__ v, float vk)
{
	const float vu = (n.n_up >= 0) ? __ldcg(v + n.n_up) : 0.f;
	const float vl = (n.n_left >= 0) ? __ldcg(v + n.n_left) : 0.f;
	const float vd = (n.n_down >= 0) ? __ldcg(v + n.n_down) : 0.f;
	const float vr = (n.n_right >= 0) ? __ldcg(v + n.n_right) : 0.f;
	const float sum = n.s_up + n.s_left + n.s_down + n.s_right;
	const float lap = n.s_up * vu + n.s_left * vl + n.s_down * vd + n.s_right * vr - vk * sum;
	return lam * n.S * vk - (1.0f - lam) * lap;
}

constexpr int kCgBlock = 512;

// Deterministic grid reduction of the first nv of 8 values per block:
// every block sums the per-block partials in the same order, so all blocks
// see identical totals.
__device__ __forceinline__ void reduce_partials(const double *__restrict__ part, int nblocks, int nv, double *out,
                                                double *smem)
{
	const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
	if (wid < nv) {
		double v = 0.0;
		for (int b = lane; b < nblocks; b += 32) v += __ldcg(part + (size_t)b * 8 + wid);
		v = warp_sum(v);
		if (lane == 0) smem[wid] = v;
	}
	__syncthreads();
	for (int c = 0; c < nv; c++) out[c] = smem[c];
	__syncthreads();
}

// Jacobi preconditioner of a row of the grid kernel's system (see
// jacobi_inv of the cluster kernel).
__device__ __forceinline__ float jacobi_inv_grid(const Unknown &n, float lam)
{
	const float dg = lam * n.S + (1.0f - lam) * (n.s_up + n.s_left + n.s_down + n.s_right);
	return (dg > 0.f) ? 1.0f / dg : 1.0f;
}

// The solver of systems larger than the SMs hold (see k_poisson_cg_wide).
// Conjugate gradient of conjugte_gradient (:387-477) for all channels at
// once: r = b - A x0, d = r; per iteration q = A d, alpha = |r|^2 / <r,q>,
// x += alpha d, r -= alpha q, beta = |r_new|^2 / |r|^2, d = r + beta d; a
// channel stops when |r|^2 < tol |r0|^2 or after `limit` iterations.
// Vectors are float, inner products double.  The grid is co-resident
// (cooperative launch) and phases are separated by the bounded barrier.
// Ends by writing u = orig + x into the image and the partial sums of
// (u_old - u_new)^2.  PRE: Jacobi-preconditioned as the cluster kernel
// (z = M r kept in `z`, d = z + beta d, alpha = <r, z> / <z, q>), same
// stopping test.
template <bool PRE>
__global__ void __launch_bounds__(kCgBlock) k_poisson_cg(PoissonArgs a, const Unknown *__restrict__ unk,
                                                         const float *__restrict__ b, float *__restrict__ x,
                                                         float *__restrict__ r, float *__restrict__ d,
                                                         float *__restrict__ q, float *__restrict__ z,
                                                         double *__restrict__ part, DevStatus *st,
                                                         int *__restrict__ iters_out,
                                                         const int32_t *__restrict__ hole,
                                                         const float *orig, float *img,
                                                         double *__restrict__ diff_part,
                                                         const int *__restrict__ active_flag)
{
	// a batch image that has stopped iterating: every block leaves at once
	if (active_flag && *active_flag == 0) return;
	__shared__ double red[kCgBlock / 32][8];
	__shared__ double tot[8];
	const int nh = a.nh, C = a.C;
	const int NV = PRE ? 2 * C : C;  // sums of the residual phase: |r|^2 (and <r, z>)
	const unsigned nb = gridDim.x;
	const int stride = gridDim.x * blockDim.x;
	double *partA = part;                   // [nb][8]
	double *partB = part + (size_t)nb * 8;  // [nb][8]
	if (!PRE) z = r;

	auto block_partial = [&](double *v, double *dst, int nv) {
		// v[nv] per thread -> dst[blockIdx.x][c]
		const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
		for (int c = 0; c < nv; c++) {
			double s = warp_sum(v[c]);
			if (lane == 0) red[wid][c] = s;
		}
		__syncthreads();
		if (threadIdx.x < nv) {
			double s = 0.0;
			for (int w = 0; w < kCgBlock / 32; w++) s += red[w][threadIdx.x];
			__stcg(dst + (size_t)blockIdx.x * 8 + threadIdx.x, s);
		}
		__syncthreads();
	};

	// r = b - A x0 ; z = M r ; d = z ; |r0|^2 (and <r0, z0>)
	double acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
	for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nh; k += stride) {
		const Unknown n = unk[k];
		for (int c = 0; c < C; c++) {
			const float *xc = x + (size_t)c * nh;
			const float rv = b[(size_t)c * nh + k] - apply_A(n, a.lambda[c], xc, __ldcg(xc + k));
			__stcg(r + (size_t)c * nh + k, rv);
			acc[c] += (double)rv * rv;
			float zv = rv;
			if (PRE) {
				zv = jacobi_inv_grid(n, a.lambda[c]) * rv;
				__stcg(z + (size_t)c * nh + k, zv);
				acc[C + c] += (double)rv * zv;
			}
			__stcg(d + (size_t)c * nh + k, zv);
		}
	}
	block_partial(acc, partB, NV);
	if (!grid_barrier(st, nb)) return;
	double nr0[4], nr[4], rho[4], t8[8];
	reduce_partials(partB, nb, NV, t8, &tot[0]);
	bool active[4];
	int it[4];
	for (int c = 0; c < 4; c++) {
		nr0[c] = (c < C) ? t8[c] : 0.0;
		nr[c] = nr0[c];
		rho[c] = (c < C) ? (PRE ? t8[C + c] : t8[c]) : 0.0;
		active[c] = (c < C) && (nr0[c] > 0);
		it[c] = 0;
	}
	for (;;) {
		bool any = false;
		for (int c = 0; c < C; c++) any |= active[c];
		if (!any) break;
		// q = A d ; <z, q>
		for (int c = 0; c < 8; c++) acc[c] = 0.0;
		for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nh; k += stride) {
			const Unknown n = unk[k];
			for (int c = 0; c < C; c++) {
				if (!active[c]) continue;
				const float *dc = d + (size_t)c * nh;
				const float qv = apply_A(n, a.lambda[c], dc, __ldcg(dc + k));
				__stcg(q + (size_t)c * nh + k, qv);
				acc[c] += (double)__ldcg(z + (size_t)c * nh + k) * qv;
			}
		}
		block_partial(acc, partA, C);
		if (!grid_barrier(st, nb)) return;
		double rq[8];
		reduce_partials(partA, nb, C, rq, &tot[0]);
		float alpha[4];
		for (int c = 0; c < C; c++) alpha[c] = active[c] ? (float)(rho[c] / rq[c]) : 0.f;
		// x += alpha d ; r -= alpha q ; z = M r ; |r|^2 (and <r, z>)
		for (int c = 0; c < 8; c++) acc[c] = 0.0;
		for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nh; k += stride) {
			Unknown n;
			if (PRE) n = unk[k];
			for (int c = 0; c < C; c++) {
				if (!active[c]) continue;
				const size_t o = (size_t)c * nh + k;
				const float dv = __ldcg(d + o);
				__stcg(x + o, __ldcg(x + o) + alpha[c] * dv);
				const float rv = __ldcg(r + o) - alpha[c] * __ldcg(q + o);
				__stcg(r + o, rv);
				acc[c] += (double)rv * rv;
				if (PRE) {
					const float zv = jacobi_inv_grid(n, a.lambda[c]) * rv;
					__stcg(z + o, zv);
					acc[C + c] += (double)rv * zv;
				}
			}
		}
		block_partial(acc, partB, NV);
		if (!grid_barrier(st, nb)) return;
		double nrn[8];
		reduce_partials(partB, nb, NV, nrn, &tot[0]);
		float beta[4];
		for (int c = 0; c < C; c++) {
			const double rhon = PRE ? nrn[C + c] : nrn[c];
			beta[c] = active[c] ? (float)(rhon / rho[c]) : 0.f;
			if (active[c]) {
				nr[c] = nrn[c];
				rho[c] = rhon;
			}
		}
		// d = z + beta d
		for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nh; k += stride) {
			for (int c = 0; c < C; c++) {
				if (!active[c]) continue;
				const size_t o = (size_t)c * nh + k;
				__stcg(d + o, __ldcg(z + o) + beta[c] * __ldcg(d + o));
			}
		}
		for (int c = 0; c < C; c++) {
			if (!active[c]) continue;
			const bool stop = (nr[c] < (double)a.tol * nr0[c]) || (it[c] >= a.limit);
			it[c]++;
			if (stop) active[c] = false;
		}
		if (!grid_barrier(st, nb)) return;
	}
	if (blockIdx.x == 0 && threadIdx.x < C) iters_out[threadIdx.x] = it[threadIdx.x];
	// u = orig + delta on the hole (:89-104)
	double dacc = 0.0;
	for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nh; k += stride) {
		const int pix = hole[k];
		for (int c = 0; c < C; c++) {
			const float o = orig[(size_t)C * pix + c];
			const float v = o + __ldcg(x + (size_t)c * nh + k);
			const float prev = img[(size_t)C * pix + c];
			const float dd = prev - v;
			dacc += (double)(dd * dd);
			img[(size_t)C * pix + c] = v;
		}
	}
	dacc = block_sum<kCgBlock>(dacc, &red[0][0]);
	if (threadIdx.x == 0) diff_part[blockIdx.x] = dacc;
}

// Conjugate gradient on thread-block clusters with the vectors in registers
// and shared memory.  Cluster g of the grid solves channel g of the image;
// the channels are independent systems (the reference solves them one
// after the other), so one cluster per channel spreads the solve over more
// SMs and lets each channel stop at its own convergence.
//
// CTA `rank` of the cluster (up to 16 CTAs of 512 threads) owns the
// contiguous unknown range [rank * chunk, (rank + 1) * chunk), chunk <= 4096;
// thread t of it owns unknowns t, t + 512, ... and keeps their rows of the
// system, r, x, d and q in registers.  Iteration (as the reference's
// conjugte_gradient, patch_non_local_poisson.cpp:387-477, with the residual
// updated by recurrence): d = r + beta d_old (folded into the stencil phase,
// formed at the neighbours from r and d_old), q = A d, alpha = |r|^2 / <r, q>,
// x += alpha d, r -= alpha q, beta = |r'|^2 / |r|^2.
//
// What a neighbour needs, the pair (r, d), is one float2 in shared memory, in
// two alternating buffers: the update phase writes the new pair of every own
// unknown with one store, and pushes it to the CTAs that have a neighbour of
// it (the first and last pixel rows of a range), which hold a slot per such
// neighbour; so the stencil reads four local float2 and nothing remote.
//
// An iteration is two exchanges between the CTAs and little else: everything
// that crosses goes by asynchronous stores that complete on the receiver's
// mbarrier, which warp 0 waits on.  At 16 CTAs, in cycles: exchanging one sum
// per CTA so takes 449 (both block barriers included), with 512 pairs pushed
// as well 745; a cluster barrier alone takes 522 (its release fence: 137
// without), plain remote stores and a cluster barrier 1278, remote loads
// instead of pushes 1373, and every warp pushing its own sum 2233.
//
// The sums.  Per thread in float, per warp in float, then in double over the
// CTA's warps and over the CTAs, and alpha and beta are rounded quotients of
// two such sums.  FP64 is slow here (62 cycles an addition, 562 a division: 1400
// per exchange in its dependent chain), so what is formed is the sum as an
// unevaluated pair of floats (Knuth's two-sum), exact to 2^-43, and the quotient
// as such a pair.  Where every value within its error bound rounds to the same
// float, that float is the quotient of the double sums; in the few cases
// where it is not (about one in 16 000, and sums outside 1e-18 .. 1e18) the double
// sums are formed (cg_double_total).  So are the stopping test's.
//
// 512 x 512 (39 000 unknowns, 3 x 16 CTAs, 73 iterations a channel, ncu): 185
// us, 2.3 us an iteration, bound by the two exchanges and the block barriers
// around them; 472 us with the rows and vectors in shared memory, remote
// loads, two cluster barriers and double sums.
constexpr int kClusterBlock = 512;
constexpr int kClusterMax = 16;
constexpr int kClusterMaxChunk = 4096;
constexpr int kClusterPerThread = kClusterMaxChunk / kClusterBlock;  // unknowns per thread

// 1 / the diagonal of an unknown's row, lam S + (1 - lam) (sum of its four
// link coefficients) (1 where that is not positive): the Jacobi
// preconditioner of the PRE kernels.
__device__ __forceinline__ float jacobi_inv(const UnkC &n, float lam)
{
	const float sum = n.s_up + n.s_left + ((n.links & 1) ? n.S : 0.f) + ((n.links & 2) ? n.S : 0.f);
	const float dg = lam * n.S + (1.0f - lam) * sum;
	return (dg > 0.f) ? 1.0f / dg : 1.0f;
}

// PRE: Jacobi-preconditioned CG (NLI_TUNE_CG_PRECOND): z = M r with M the
// inverse diagonal, d = z + beta d_old, alpha = <r, z> / <z, A d>, beta =
// <r', z'> / <r, z>.  The stopping test stays |r|^2 < tol |r0|^2 on the
// true residual, so the solve ends at the same residual as the plain CG,
// in fewer iterations.  Without PRE, z is r itself and the iteration is the
// reference's.
// Slots of a buffer of (r, d) pairs for ranges of `chunk` unknowns: the own
// unknowns, then for each the slot of its upper and of its lower neighbour
// where another CTA owns it, those of the range's left and right neighbour,
// and one that stays zero for neighbours outside the hole.
__host__ __device__ inline int cg_slots(int chunk) { return 3 * chunk + 3; }

__host__ inline size_t cg_smem_bytes(int chunk) { return 2 * sizeof(float2) * (size_t)cg_slots(chunk); }

// A sum as an unevaluated pair h + l, with the sum of its terms' magnitudes
// (what its error is measured by: below 2^-43 a).
struct Sum2 {
	float h, l, a;
};

__device__ __forceinline__ Sum2 sum2(float v) { return {v, 0.f, fabsf(v)}; }

__device__ __forceinline__ Sum2 sum2_add(Sum2 x, Sum2 y)
{
	const float s = x.h + y.h, t = s - x.h;
	float e = (x.h - (s - t)) + (y.h - t);  // exact (two-sum)
	e += x.l + y.l;
	const float h = s + e;
	return {h, e - (h - s), x.a + y.a};
}

__device__ __forceinline__ Sum2 sum2_shfl(Sum2 x, int o)
{
	return {__shfl_xor_sync(0xffffffffu, x.h, o), __shfl_xor_sync(0xffffffffu, x.l, o),
	        __shfl_xor_sync(0xffffffffu, x.a, o)};
}

// The sum over 16 lanes, of which the warp's halves hold the same: every lane
// of the warp ends with the same total.
__device__ __forceinline__ Sum2 sum2_16(Sum2 x)
{
#pragma unroll
	for (int o = 8; o > 0; o >>= 1) x = sum2_add(x, sum2_shfl(x, o));
	return x;
}

// Bounds of what the pair arithmetic takes: nothing in it can over- or
// underflow.
__device__ __forceinline__ bool sum2_safe(float v) { return fabsf(v) >= 1e-18f && fabsf(v) <= 1e18f; }

// float(n / d) of the double sums that n and d approximate; false where the
// pairs do not decide it.
__device__ __forceinline__ bool sum2_quotient(Sum2 n, Sum2 d, float &q)
{
	const float y = __fdividef(1.0f, d.h);
	const float q0 = n.h * y;
	const float rem = fmaf(-q0, d.l, fmaf(-q0, d.h, n.h) + n.l);
	const float q1 = rem * y;
	const float m = fabsf(q0) * 0x1p-40f * (2.0f + d.a * fabsf(y));
	const float lo = q0 + (q1 - m), hi = q0 + (q1 + m);
	q = lo;
	return lo == hi && sum2_safe(n.h) && sum2_safe(d.h) && sum2_safe(q0) && d.a <= 1e18f;
}

__device__ __forceinline__ uint32_t cg_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ uint32_t cg_remote(uint32_t addr, int rank)
{
	uint32_t a;
	asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(addr), "r"(rank));
	return a;
}

// Asynchronous stores into a CTA of the cluster (addresses from cg_remote)
// that complete on its mbarrier.
__device__ __forceinline__ void cg_send(uint32_t dst, float2 v, uint32_t bar)
{
	asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.f32 [%0], {%1, %2}, [%3];" ::"r"(dst),
	             "f"(v.x), "f"(v.y), "r"(bar)
	             : "memory");
}

__device__ __forceinline__ void cg_send(uint32_t dst, float4 v, uint32_t bar)
{
	asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(dst),
	             "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w), "r"(bar)
	             : "memory");
}

__device__ __forceinline__ void cg_send(uint32_t dst, double v, uint32_t bar)
{
	asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(dst),
	             "l"(__double_as_longlong(v)), "r"(bar)
	             : "memory");
}

// One arrival and `bytes` to come for the barrier's current phase.
__device__ __forceinline__ void cg_expect(uint32_t bar, uint32_t bytes)
{
	asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}

// Waits for phase `parity`; false when the bounded wait ran out (each poll
// suspends for a microsecond at most: about a second in all).
__device__ __forceinline__ bool cg_wait(uint32_t bar, uint32_t parity)
{
	constexpr uint32_t kPolls = 1u << 20, kPollNs = 1000u;
	uint32_t ok = 0;
	for (uint32_t i = 0; i < kPolls && !ok; i++)
		asm volatile(
		    "{\n\t.reg .pred p;\n\t"
		    "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2, %3;\n\t"
		    "selp.u32 %0, 1, 0, p;\n\t}"
		    : "=r"(ok)
		    : "r"(bar), "r"(parity), "r"(kPollNs)
		    : "memory");
	return ok != 0;
}

// Shared memory of a solve beside the pairs.
enum CgBar { kBarStencil = 0, kBarUpdate = 1, kBarDouble = 2 };

template <bool PRE>
struct CgShared {
	static constexpr int NV = PRE ? 2 : 1;  // sums of the update phase: |r|^2 (and <r, z>)
	float4 sumA[kClusterMax], sumB[NV][kClusterMax];  // every CTA's, by rank
	double dbl[2][kClusterMax];
	uint64_t bar[3];
	float redA[16], redB[2][NV][16];  // this CTA's warps'; the update phase's last two
	double red[kClusterBlock / 32];
	float coef;
	int active, ghosts;
	uint32_t doubles;  // exchanges on kBarDouble so far
	int failed;        // a wait ran out
};

// The sum over the cluster in double, of warp sums red (16 per CTA): per CTA a
// shuffle tree over its warps, then one over the CTAs.  Called by warp 0 of
// every CTA alike; every lane returns the total.
template <bool PRE, bool SINGLE>
__device__ __noinline__ double cg_double_total(CgShared<PRE> &sh, const float *red, int rank, int ncta)
{
	const int lane = threadIdx.x & 31;
	double v = warp_sum(lane < 16 ? (double)red[lane] : 0.0);
	v = __shfl_sync(0xffffffffu, v, 0);
	if (SINGLE) return v;
	const uint32_t n = sh.doubles, bar = cg_u32(&sh.bar[kBarDouble]);
	__syncwarp();
	if (lane < ncta) cg_send(cg_remote(cg_u32(&sh.dbl[n & 1][rank]), lane), v, cg_remote(bar, lane));
	const bool ok = __all_sync(0xffffffffu, cg_wait(bar, n & 1));
	if (lane == 0) {
		cg_expect(bar, ncta * (uint32_t)sizeof(double));
		sh.doubles = n + 1;
		if (!ok) sh.failed = 1;
	}
	__syncwarp();
	v = warp_sum(lane < ncta ? sh.dbl[n & 1][lane] : 0.0);
	return __shfl_sync(0xffffffffu, v, 0);
}

// The solve of channel ch of the a.C-channel image by a cluster's CTAs, or by
// one CTA on its own (SINGLE; the arithmetic of a cluster of one); U: unknowns
// per thread at most; timeout: the context's status word.
template <bool PRE, bool SINGLE, int U>
__device__ __forceinline__ void cg_team_solve(const PoissonArgs &a, int chunk, const UnkC *__restrict__ unk_g,
                                              const float *__restrict__ b, const float *__restrict__ x0,
                                              int *__restrict__ iters_out, const int32_t *__restrict__ hole,
                                              const float *orig, float *img, double *__restrict__ diff_part, int ch,
                                              int *timeout)
{
	extern __shared__ float2 s_pair[];  // two buffers of cg_slots(chunk)
	__shared__ __align__(16) CgShared<PRE> sh;
	constexpr int NV = PRE ? 2 : 1;
	int rank = 0, ncta = 1;
	if (!SINGLE) {
		rank = (int)cooperative_groups::this_cluster().block_rank();
		ncta = (int)cooperative_groups::this_cluster().num_blocks();
	}
	const int Ctot = a.C, nh = a.nh;
	b += (size_t)ch * nh;
	x0 += (size_t)ch * nh;
	const int lo = rank * chunk, own = max(0, min(nh, lo + chunk) - lo);
	const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
	const int slots = cg_slots(chunk), zero_slot = 3 * chunk + 2;
	const float oml = 1.0f - a.lambda[ch];
	const uint32_t bar_a = cg_u32(&sh.bar[kBarStencil]), bar_b = cg_u32(&sh.bar[kBarUpdate]);

	if (threadIdx.x == 0) {
		sh.ghosts = 0;
		sh.doubles = 0;
		sh.failed = 0;
		if (!SINGLE) {
			for (int i = 0; i < 3; i++)
				asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(cg_u32(&sh.bar[i])) : "memory");
			asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
		}
	}
	if (threadIdx.x < 2) s_pair[threadIdx.x * slots + zero_slot] = make_float2(0.f, 0.f);
	__syncthreads();

	// this thread's unknowns: the row (up and left link, own coefficient, sum of
	// the links, lambda S), the neighbours' slots (up | down << 16, left |
	// right << 16) and for those of other CTAs their codes (owner << 12 | index)
	float su[U], sl[U], sc[U], sum[U], ls[U], minv[PRE ? U : 1];
	uint32_t nud[U], nlr[U], cud[U], clr[U];
	float r[U], x[U], d[U], q[U];
	float acc = 0.f, accz = 0.f;
	int ghosts = 0;
	// r0 = b - A x0 (x0 from global: neighbours may belong to other CTAs)
#pragma unroll
	for (int u = 0; u < U; u++) {
		const int l = threadIdx.x + u * kClusterBlock;
		if (l >= own) break;
		const int k = lo + l;
		const UnkC n = unk_g[k];
		const uint32_t codes[4] = {n.ud >> 16, n.lr >> 16, n.ud & 0xFFFF, n.lr & 0xFFFF};
		const float coefs[4] = {n.s_up, n.s_left, (n.links & 1) ? n.S : 0.f, (n.links & 2) ? n.S : 0.f};
		const float sm = coefs[0] + coefs[1] + coefs[2] + coefs[3];
		int gk[4], slot[4];
		uint32_t far[4];
#pragma unroll
		for (int j = 0; j < 4; j++) {
			gk[j] = (codes[j] != kNoNb) ? (int)(codes[j] >> 12) * chunk + (int)(codes[j] & 0xFFF) : -1;
			if (gk[j] >= 0 && !nli_in_bounds(gk[j], nh, kSiteCgNeighbour)) gk[j] = -1;
			const bool local = gk[j] >= 0 && (int)(codes[j] >> 12) == rank;
			far[j] = gk[j] >= 0 && !local ? codes[j] : (uint32_t)kNoNb;
			ghosts += far[j] != kNoNb;
			slot[j] = gk[j] < 0 ? zero_slot
			          : local   ? (int)(codes[j] & 0xFFF)
			          : j == 0  ? chunk + l
			          : j == 2  ? 2 * chunk + l
			          : j == 1  ? 3 * chunk
			                    : 3 * chunk + 1;
		}
		su[u] = n.s_up;
		sl[u] = n.s_left;
		sc[u] = n.S;
		sum[u] = sm;
		ls[u] = a.lambda[ch] * n.S;
		nud[u] = (uint32_t)slot[0] | ((uint32_t)slot[2] << 16);
		nlr[u] = (uint32_t)slot[1] | ((uint32_t)slot[3] << 16);
		cud[u] = far[0] | (far[2] << 16);
		clr[u] = far[1] | (far[3] << 16);
		const float xk = x0[k];
		float lap = -xk * sm;
#pragma unroll
		for (int j = 0; j < 4; j++)
			if (gk[j] >= 0) lap += coefs[j] * x0[gk[j]];
		const float rv = b[k] - (a.lambda[ch] * n.S * xk - (1.0f - a.lambda[ch]) * lap);
		r[u] = rv;
		x[u] = xk;
		d[u] = 0.f;
		acc = fmaf(rv, rv, acc);
		if (PRE) {
			minv[u] = jacobi_inv(n, a.lambda[ch]);
			accz = fmaf(rv, fm(minv[u], rv), accz);
		}
	}
	if (!SINGLE && ghosts) atomicAdd(&sh.ghosts, ghosts);
	__syncthreads();
	// bytes an update phase brings: every CTA's sums and a pair per neighbour of
	// an own unknown that another CTA owns (which has this one as neighbour)
	const uint32_t bytes_a = ncta * (uint32_t)sizeof(float4);
	const uint32_t bytes_b = NV * bytes_a + sh.ghosts * (uint32_t)sizeof(float2);
	if (!SINGLE) {
		if (threadIdx.x == 0) {
			cg_expect(bar_a, bytes_a);
			cg_expect(bar_b, bytes_b);
			cg_expect(cg_u32(&sh.bar[kBarDouble]), ncta * (uint32_t)sizeof(double));
		}
		// every CTA's barriers are ready before anything is sent
		cooperative_groups::this_cluster().sync();
	}

	// the pair of every own unknown into buffer h, and into the slots of the
	// CTAs that have it as a neighbour: it is its upper neighbour's lower
	// neighbour, and so on
	auto publish = [&](int h) {
		float2 *buf = s_pair + h * slots;
#pragma unroll
		for (int u = 0; u < U; u++) {
			const int l = threadIdx.x + u * kClusterBlock;
			if (l >= own) break;
			const float2 v = make_float2(PRE ? fm(minv[u], r[u]) : r[u], d[u]);
			buf[l] = v;
			if (SINGLE || (cud[u] & clr[u]) == 0xffffffffu) continue;
			auto push = [&](uint32_t code, int slot) {
				if (code == (uint32_t)kNoNb) return;
				const int to = (int)(code >> 12);
				cg_send(cg_remote(cg_u32(buf + slot), to), v, cg_remote(bar_b, to));
			};
			push(cud[u] & 0xFFFF, 2 * chunk + (int)(cud[u] & 0xFFF));
			push(cud[u] >> 16, chunk + (int)((cud[u] >> 16) & 0xFFF));
			push(clr[u] & 0xFFFF, 3 * chunk + 1);
			push(clr[u] >> 16, 3 * chunk);
		}
	};
	// warp 0, after a block barrier: the CTA's sum of red sent to every CTA
	auto send_sum = [&](const float *red, float4 *dst, uint32_t bar) {
		const Sum2 t = sum2_16(sum2(red[lane & 15]));
		const float4 v = make_float4(t.h, t.l, t.a, 0.f);
		if (SINGLE) {
			if (lane == 0) dst[0] = v;
			__syncwarp();
		} else if (lane < ncta) {
			cg_send(cg_remote(cg_u32(dst + rank), lane), v, cg_remote(bar, lane));
		}
	};
	auto wait = [&](uint32_t bar, uint32_t parity, uint32_t bytes) {
		if (SINGLE) return;
		const bool ok = __all_sync(0xffffffffu, cg_wait(bar, parity));
		if (lane == 0) {
			cg_expect(bar, bytes);
			if (!ok) sh.failed = 1;
		}
		__syncwarp();
	};
	auto total = [&](const float4 *src) {
		const float4 v = (lane & 15) < ncta ? src[lane & 15] : make_float4(0.f, 0.f, 0.f, 0.f);
		return sum2_16(Sum2{v.x, v.y, v.z});
	};

	publish(0);
	acc = warp_sum(acc);
	accz = PRE ? warp_sum(accz) : 0.f;
	if (lane == 0) {
		sh.redB[0][0][wid] = acc;
		if (PRE) sh.redB[0][NV - 1][wid] = accz;
	}
	__syncthreads();
	// warp 0 holds the solve's scalars
	Sum2 rho = sum2(0.f), stop = sum2(0.f);  // <r, z>; tol |r0|^2
	double nr0 = 0.0;
	int it = 0;
	uint32_t parity = 0;  // of the phases of bar_a (and, one ahead, of bar_b)
	if (wid == 0) {
		for (int v = 0; v < NV; v++) send_sum(sh.redB[0][v], sh.sumB[v], bar_b);
		wait(bar_b, 0, bytes_b);
		rho = total(sh.sumB[NV - 1]);
		nr0 = cg_double_total<PRE, SINGLE>(sh, sh.redB[0][0], rank, ncta);
		const double t = (double)a.tol * nr0;
		stop.h = (float)t;
		stop.l = (float)(t - (double)stop.h);
		stop.a = fabsf(stop.h);
		if (lane == 0) sh.active = nr0 > 0 && !sh.failed;
	}
	__syncthreads();
	bool active = sh.active != 0;
	float beta = 0.f;
	int h = 0;  // buffer of the current pairs
	while (active) {
		// d = z + beta d_old (own and neighbours) ; q = A d ; <z, q>
		const float2 *buf = s_pair + h * slots;
		acc = 0.f;
#pragma unroll
		for (int u = 0; u < U; u++) {
			if ((int)threadIdx.x + u * kClusterBlock >= own) break;
			const float2 vu = buf[nud[u] & 0xFFFF], vl = buf[nlr[u] & 0xFFFF];
			const float2 vd = buf[nud[u] >> 16], vr = buf[nlr[u] >> 16];
			const float rk = PRE ? fm(minv[u], r[u]) : r[u];
			const float dk = fmaf(beta, d[u], rk);
			// a neighbour outside the hole reads zeros
			float lap = fm(-dk, sum[u]);
			lap = fmaf(su[u], fmaf(beta, vu.y, vu.x), lap);
			lap = fmaf(sl[u], fmaf(beta, vl.y, vl.x), lap);
			lap = fmaf(sc[u], fmaf(beta, vd.y, vd.x), lap);
			lap = fmaf(sc[u], fmaf(beta, vr.y, vr.x), lap);
			const float qv = fmaf(ls[u], dk, -fm(oml, lap));
			d[u] = dk;
			q[u] = qv;
			acc = fmaf(rk, qv, acc);
		}
		acc = warp_sum(acc);
		if (lane == 0) sh.redA[wid] = acc;
		__syncthreads();
		if (wid == 0) {
			send_sum(sh.redA, sh.sumA, bar_a);
			wait(bar_a, parity, bytes_a);
			float alpha;
			if (!sum2_quotient(rho, total(sh.sumA), alpha)) {
				const double rq = cg_double_total<PRE, SINGLE>(sh, sh.redA, rank, ncta);
				alpha = (float)(cg_double_total<PRE, SINGLE>(sh, sh.redB[h][NV - 1], rank, ncta) / rq);
			}
			if (lane == 0) sh.coef = alpha;
		}
		__syncthreads();
		const float alpha = sh.coef;
		// r -= alpha q ; z = M r ; |r|^2 (and <r, z>) ; x += alpha d
		acc = accz = 0.f;
#pragma unroll
		for (int u = 0; u < U; u++) {
			if ((int)threadIdx.x + u * kClusterBlock >= own) break;
			r[u] = fmaf(-alpha, q[u], r[u]);
			acc = fmaf(r[u], r[u], acc);
			if (PRE) accz = fmaf(r[u], fm(minv[u], r[u]), accz);
		}
		h = 1 - h;
		publish(h);
		acc = warp_sum(acc);
		accz = PRE ? warp_sum(accz) : 0.f;
		if (lane == 0) {
			sh.redB[h][0][wid] = acc;
			if (PRE) sh.redB[h][NV - 1][wid] = accz;
		}
		__syncthreads();
		if (wid == 0) {
			for (int v = 0; v < NV; v++) send_sum(sh.redB[h][v], sh.sumB[v], bar_b);
			wait(bar_b, parity ^ 1u, bytes_b);
			const Sum2 nrn = total(sh.sumB[0]), rhon = PRE ? total(sh.sumB[NV - 1]) : nrn;
			float bt;
			const float over = (nrn.h - stop.h) + (nrn.l - stop.l);
			bool done = over < 0.f;
			if (!sum2_quotient(rhon, rho, bt) || !sum2_safe(nrn.h) ||
			    !(fabsf(over) > 0x1p-39f * (nrn.a + stop.a))) {
				const double rn = cg_double_total<PRE, SINGLE>(sh, sh.redB[h][0], rank, ncta);
				const double zn = PRE ? cg_double_total<PRE, SINGLE>(sh, sh.redB[h][NV - 1], rank, ncta) : rn;
				bt = (float)(zn / cg_double_total<PRE, SINGLE>(sh, sh.redB[1 - h][NV - 1], rank, ncta));
				done = rn < (double)a.tol * nr0;
			}
			if (lane == 0) {
				sh.coef = bt;
				sh.active = !(done || it >= a.limit || sh.failed);
			}
			rho = rhon;
			it++;
		}
#pragma unroll
		for (int u = 0; u < U; u++) {
			if ((int)threadIdx.x + u * kClusterBlock >= own) break;
			x[u] = fmaf(alpha, d[u], x[u]);
		}
		parity ^= 1u;
		// the sums of a phase arrive again only after the other phase, in which
		// every warp 0 has read them; coef and active change only after the
		// next block barrier, by which every thread has
		__syncthreads();
		beta = sh.coef;
		active = sh.active != 0;
	}
	if (rank == 0 && threadIdx.x == 0) iters_out[ch] = it;
	if (threadIdx.x == 0 && sh.failed) {
		// the missing data may still land: one more bounded wait before leaving
		cg_wait(bar_a, parity);
		cg_wait(bar_b, parity ^ 1u);
		atomicExch(timeout, 1);
	}
	// u = orig + delta on the hole (:89-104)
	double dacc = 0.0;
#pragma unroll
	for (int u = 0; u < U; u++) {
		const int l = threadIdx.x + u * kClusterBlock;
		if (l >= own) break;
		const int pix = hole[lo + l];
		const float o = orig[(size_t)Ctot * pix + ch];
		const float v = o + x[u];
		const float prev = img[(size_t)Ctot * pix + ch];
		const float dd = prev - v;
		dacc += (double)(dd * dd);
		img[(size_t)Ctot * pix + ch] = v;
	}
	dacc = block_sum<kClusterBlock>(dacc, sh.red);
	if (threadIdx.x == 0) diff_part[ch * ncta + rank] = dacc;
	// no CTA leaves while one may still send to it
	if (!SINGLE) cooperative_groups::this_cluster().sync();
}

// Unknowns per thread the solvers are compiled for.  The arrays of unused ones cost
// time: an update whose CTAs hold 1024 unknowns takes 184 us with 2, 3 or 5 per thread
// and 207 with 8, with 2048 unknowns 207 us with 4, 210 with 5 and 236 with 8, with 2430
// (a 512 x 512 image's 39 000) 222 with 5, 229 with 6 and 254 with 8.  Above, 6 and 7 where they suffice
// would gain too (3000 unknowns: 242, 263 and 268 us with 6, 7 and 8; 3480: 280
// and 297 with 7 and 8), at six more kernels for each count.  k_poisson_cg_wide:
// 1390 unknowns 365 us with 3, 360 with 4, 377 with 5, 510 with 8; 2500 unknowns 640 us with 5
// and with 8; 3000: 728 with 6, 760 with 7 and 8; 3500: 685 with 7, 694 with 8.
constexpr int cg_per_thread(int chunk)
{
	return chunk <= 2 * kClusterBlock ? 2 : chunk <= 5 * kClusterBlock ? 5 : kClusterPerThread;
}

template <bool PRE, int U>
__global__ void __launch_bounds__(kClusterBlock, 1)
    k_poisson_cg_cluster(PoissonArgs a, int chunk, const UnkC *__restrict__ unk_g, const float *__restrict__ b,
                         const float *__restrict__ x0, int *__restrict__ iters_out, const int32_t *__restrict__ hole,
                         const float *orig, float *img, double *__restrict__ diff_part, int *timeout)
{
	const int ncta = (int)cooperative_groups::this_cluster().num_blocks();
	cg_team_solve<PRE, false, U>(a, chunk, unk_g, b, x0, iters_out, hole, orig, img, diff_part,
	                             (int)blockIdx.x / ncta, timeout);
}

// One CTA per channel (systems of at most kClusterMaxChunk unknowns).
template <bool PRE, int U>
__global__ void __launch_bounds__(kClusterBlock, 1)
    k_poisson_cg_cta(PoissonArgs a, int chunk, const UnkC *__restrict__ unk_g, const float *__restrict__ b,
                     const float *__restrict__ x0, int *__restrict__ iters_out, const int32_t *__restrict__ hole,
                     const float *orig, float *img, double *__restrict__ diff_part, int *timeout)
{
	cg_team_solve<PRE, true, U>(a, chunk, unk_g, b, x0, iters_out, hole, orig, img, diff_part, (int)blockIdx.x,
	                            timeout);
}

// ------------------------------------------------ CG over the whole grid
// Systems too large for a cluster: the cluster CG's scheme with its CTAs on
// every SM and the exchanges through L2.  A group of `ctas` CTAs solves one
// channel, up to C groups side by side (a cooperative launch: all are
// resident); each CTA owns a contiguous range of at most 4096 unknowns whose
// rows and vectors stay in its registers and shared memory.
//
// What crosses: the (r, d) pair of an unknown with a neighbour in another
// range, and each CTA's sums.  A value travels in a 64-bit word with the
// number of its exchange in the upper half, stored and polled with relaxed
// accesses: data and flag arrive as one, so nothing is fenced, no barrier is
// taken, and a CTA waits for exactly what it reads: warp 0 for the sums (it
// holds the solve's scalars), the others meanwhile for the pairs that the
// next stencil needs, several loads in flight.  The words are cleared
// before the launch.  Pairs alternate between two buffers; sums need one per
// phase, because a CTA sends its next of a phase only after it has had every
// CTA's of the other, which they send after reading the last.
//
// The per-thread and per-CTA sums are pairs of floats (exact to 2^-43 of their
// terms' magnitudes, products included), in place of the double sums of
// k_poisson_cg.  Products of floats vanish or overflow where doubles do not
// (tiny or huge gradients, a tolerance near 0): a channel with a sum or quotient
// outside 1e-28 .. 1e28 is left as it was, and a second launch, DBL, whose blocks
// otherwise leave at once, solves it with every sum and quotient in double.  (One
// kernel that forms such sums again in double, by one more exchange, was 20 % slower
// on systems that never need it: 1680 us instead of 1400 for the update below.)
//
// 1024 x 685 (175 000 unknowns, 3 x 50 CTAs, 117 iterations a channel, ncu): 1.12
// ms, 9.6 us an iteration, of which the two exchanges take most: between 50 CTAs of
// both dies one takes 3700 to 4200 cycles on its own, between 8 neighbouring ones
// 800 to 1500; the empty launch with double sums takes 2.7 us.  k_poisson_cg, with
// three grid barriers and its vectors in L2, took 4.52 ms.  The same update (1.47
// ms) takes 2.08 ms on the image scaled by 2^-70 (all of it in doubles) and 2.63 ms by
// 2^-50 (in pairs until |r|^2 leaves the range, then again in doubles); it took 5.3
// ms with k_poisson_cg.
struct GridCgArgs {
	PoissonArgs a;
	int chunk, ctas, ch0;
	const Unknown *unk;
	const float *b, *x0;
	ulonglong2 *pairs;  // [2][groups of the launch][nh]
	ulonglong2 *sums;   // [groups of the launch][1 + NV][ctas]
	DevStatus *st;
	int *iters;
	int *redo;  // per channel: left to the launch with double sums
	const int32_t *hole;
	const float *orig;
	float *img;
	double *diff;
	const int *active;
};

// Whether a total or a quotient in pairs has lost nothing to the range of floats:
// what underflows is below 2^-149 a product, 1e-39 over all unknowns that the
// SMs hold.
__device__ __forceinline__ bool wide_safe(float v) { return fabsf(v) >= 1e-28f && fabsf(v) <= 1e28f; }

// Running sum of products as a pair.
struct Dot2 {
	float h = 0.f, l = 0.f;
	__device__ __forceinline__ void add(float a, float b)
	{
		const float p = fm(a, b), e = fmaf(a, b, -p);
		const float s = h + p, t = s - h;
		l += ((h - (s - t)) + (p - t)) + e;
		h = s;
	}
};

// A sum of the solve, as pairs (DBL false) or doubles: of a thread's products, and
// how it travels in two words.
template <bool DBL>
struct WideSum;

template <>
struct WideSum<false> {
	typedef Sum2 T;
	static __device__ __forceinline__ T of(const Dot2 &v) { return {v.h, v.l, 0.f}; }
	static __device__ __forceinline__ T of(float2 w) { return {w.x, w.y, 0.f}; }
	static __device__ __forceinline__ float2 words(T v) { return make_float2(v.h, v.l); }
	static __device__ __forceinline__ T add(T a, T b) { return sum2_add(a, b); }
	static __device__ __forceinline__ T shfl(T a, int o) { return sum2_shfl(a, o); }
	static __device__ __forceinline__ double value(T v) { return (double)v.h + (double)v.l; }
	static __device__ __forceinline__ float quotient(T n, T m)
	{
		const float y = __fdividef(1.0f, m.h), q0 = n.h * y;
		return q0 + fmaf(-q0, m.l, fmaf(-q0, m.h, n.h) + n.l) * y;
	}
	static __device__ __forceinline__ bool below(T a, T b) { return (a.h - b.h) + (a.l - b.l) < 0.f; }
	static __device__ __forceinline__ bool safe(T v) { return wide_safe(v.h); }
};

struct DotD {
	double s = 0.0;
	__device__ __forceinline__ void add(float a, float b) { s += (double)a * b; }
};

template <>
struct WideSum<true> {
	typedef double T;
	static __device__ __forceinline__ T of(const DotD &v) { return v.s; }
	static __device__ __forceinline__ T of(float2 w) { return __hiloint2double(__float_as_int(w.x), __float_as_int(w.y)); }
	static __device__ __forceinline__ float2 words(T v)
	{
		return make_float2(__int_as_float(__double2hiint(v)), __int_as_float(__double2loint(v)));
	}
	static __device__ __forceinline__ T add(T a, T b) { return a + b; }
	static __device__ __forceinline__ T shfl(T a, int o) { return __shfl_xor_sync(0xffffffffu, a, o); }
	static __device__ __forceinline__ double value(T v) { return v; }
	static __device__ __forceinline__ float quotient(T n, T m) { return (float)(n / m); }
	static __device__ __forceinline__ bool below(T a, T b) { return a < b; }
	static __device__ __forceinline__ bool safe(T) { return true; }
};

__device__ __forceinline__ void grid_put(ulonglong2 *p, float2 v, uint32_t tag)
{
	const unsigned long long t = (unsigned long long)tag << 32;
	asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(p), "l"(t | __float_as_uint(v.x)),
	             "l"(t | __float_as_uint(v.y))
	             : "memory");
}

// Polls the words p[i], i < n <= N, until all carry `tag`, the loads of a round
// in flight together; false when the bounded wait ran out (here or, told by
// the status word, elsewhere).
template <int N>
__device__ __forceinline__ bool grid_get(const ulonglong2 *const (&p)[N], int n, uint32_t tag, float2 (&v)[N],
                                         DevStatus *st, unsigned limit)
{
	for (unsigned polls = 0;; polls++) {
		unsigned long long x[N], y[N];
#pragma unroll
		for (int i = 0; i < N; i++)
			if (i < n)
				asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(x[i]), "=l"(y[i]) : "l"(p[i]) : "memory");
		bool all = true;
#pragma unroll
		for (int i = 0; i < N; i++)
			if (i < n) {
				all &= (uint32_t)(x[i] >> 32) == tag && (uint32_t)(y[i] >> 32) == tag;
				v[i] = make_float2(__uint_as_float((uint32_t)x[i]), __uint_as_float((uint32_t)y[i]));
			}
		if (all) return true;
		if (polls >= limit || ((polls & 255u) == 255u && *(volatile int *)&st->timeout)) {
			atomicExch(&st->timeout, 1);
			return false;
		}
	}
}

// How a solve goes on after an iteration.
enum { kCgDone, kCgOn, kCgUnsafe };

template <bool PRE, int U, bool DBL>
__global__ void __launch_bounds__(kClusterBlock, 1) k_poisson_cg_wide(const __grid_constant__ GridCgArgs A)
{
	// a batch image that has stopped iterating: every block leaves at once
	if (A.active && *A.active == 0) return;
	typedef WideSum<DBL> S;
	typedef typename S::T Sum;
	typedef typename std::conditional<DBL, DotD, Dot2>::type Dot;
	constexpr int NV = PRE ? 2 : 1;
	extern __shared__ float2 s_pair[];  // two buffers of cg_slots(chunk)
	__shared__ float2 s_red[NV][16];
	__shared__ double s_dbl[kClusterBlock / 32];
	__shared__ float s_coef;
	__shared__ int s_active, s_failed;
	__shared__ uint32_t s_far[32];  // of warp 0
	const int ctas = A.ctas, chunk = A.chunk;
	const int group = (int)blockIdx.x / ctas, rank = (int)blockIdx.x - group * ctas;
	const int ch = A.ch0 + group, C = A.a.C, nh = A.a.nh;
	if (DBL && !A.redo[ch]) return;
	const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
	const int lo = rank * chunk, own = max(0, min(nh, lo + chunk) - lo);
	const int slots = cg_slots(chunk), zero_slot = 3 * chunk + 2;
	const float lambda = A.a.lambda[ch], oml = 1.0f - lambda;
	const float *b = A.b + (size_t)ch * nh, *x0 = A.x0 + (size_t)ch * nh;
	const int groups = (int)gridDim.x / ctas;
	uint32_t *s_step = reinterpret_cast<uint32_t *>(s_pair + 2 * slots);  // [chunk], see below
	ulonglong2 *pairs = A.pairs + (size_t)group * nh;
	const size_t pair_stride = (size_t)groups * nh;  // between the two buffers
	ulonglong2 *sums = A.sums + (size_t)group * (1 + NV) * ctas;
	const unsigned set = *(volatile unsigned *)&A.st->wait_limit;
	const unsigned limit = set ? set : 1u << 22;  // some seconds

	if (threadIdx.x == 0) s_failed = 0;
	if (threadIdx.x < 2) s_pair[threadIdx.x * slots + zero_slot] = make_float2(0.f, 0.f);

	// this thread's unknowns: the row, the neighbours' slots, and which
	// neighbours lie in other ranges (far); the distance to the upper and
	// lower neighbour (up | down << 16) is in s_step
	float su[U], sl[U], sc[U], sum[U], ls[U], minv[PRE ? U : 1];
	uint32_t nud[U], nlr[U];
	uint32_t far = 0;  // 4 bits per unknown: up, left, down, right
	float r[U], x[U], d[U], q[U];
	Dot acc, accz;
#pragma unroll
	for (int u = 0; u < U; u++) {
		const int l = threadIdx.x + u * kClusterBlock;
		if (l >= own) break;
		const int k = lo + l;
		const Unknown n = A.unk[k];
		const int m[4] = {n.n_up, n.n_left, n.n_down, n.n_right};
		const float coefs[4] = {n.s_up, n.s_left, n.s_down, n.s_right};
		const float xk = x0[k];
		sum[u] = n.s_up + n.s_left + n.s_down + n.s_right;
		float lap = fm(-xk, sum[u]);
		int slot[4];
#pragma unroll
		for (int j = 0; j < 4; j++) {
			const bool there = m[j] >= 0 && nli_in_bounds(m[j], nh, kSiteCgNeighbour);
			const bool local = there && m[j] >= lo && m[j] < lo + own;
			if (there && !local) far |= 1u << (4 * u + j);
			if (there) lap = fmaf(coefs[j], x0[m[j]], lap);
			slot[j] = !there ? zero_slot : local ? m[j] - lo : j == 0 ? chunk + l : j == 2 ? 2 * chunk + l : 3 * chunk + (j == 3);
		}
		su[u] = n.s_up;
		sl[u] = n.s_left;
		sc[u] = n.S;
		ls[u] = fm(lambda, n.S);
		nud[u] = (uint32_t)slot[0] | ((uint32_t)slot[2] << 16);
		nlr[u] = (uint32_t)slot[1] | ((uint32_t)slot[3] << 16);
		s_step[l] = ((uint32_t)(k - n.n_up) & 0xFFFFu) | ((uint32_t)(n.n_down - k) << 16);
		const float rv = b[k] - fmaf(ls[u], xk, -fm(oml, lap));
		r[u] = rv;
		x[u] = xk;
		d[u] = 0.f;
		acc.add(rv, rv);
		if (PRE) {
			minv[u] = jacobi_inv_grid(n, lambda);
			accz.add(rv, fm(minv[u], rv));
		}
	}
	// the pair of every own unknown into buffer h, and with the exchange's number
	// for the CTAs that have it as a neighbour
	auto publish = [&](int h, uint32_t tag) {
		float2 *buf = s_pair + h * slots;
#pragma unroll
		for (int u = 0; u < U; u++) {
			const int l = threadIdx.x + u * kClusterBlock;
			if (l >= own) break;
			const float2 v = make_float2(PRE ? fm(minv[u], r[u]) : r[u], d[u]);
			buf[l] = v;
			if (far >> (4 * u) & 15u) grid_put(pairs + h * pair_stride + lo + l, v, tag);
		}
	};
	// the pairs of the neighbours in other ranges (f) of thread t's unknowns into
	// their slots, four loads in flight
	auto fetch_for = [&](int t, uint32_t f, int h, uint32_t tag) {
		float2 *buf = s_pair + h * slots;
		const ulonglong2 *from = pairs + h * pair_stride + lo;
		while (f) {
			const ulonglong2 *p[4];
			int slot[4], n = 0;
#pragma unroll
			for (int i = 0; i < 4; i++) {
				p[i] = nullptr;
				slot[i] = 0;
				if (f) {
					const int bit = __ffs(f) - 1, j = bit & 3, l = t + (bit >> 2) * kClusterBlock;
					f &= f - 1;
					const uint32_t st = s_step[l];
					p[i] = from + l + (j == 0 ? -(int)(st & 0xFFFFu) : j == 1 ? -1 : j == 2 ? (int)(st >> 16) : 1);
					slot[i] = j == 0 ? chunk + l : j == 2 ? 2 * chunk + l : 3 * chunk + (j == 3);
					n++;
				}
			}
			float2 v[4];
			if (!grid_get(p, n, tag, v, A.st, limit)) {
				s_failed = 1;
				return;
			}
#pragma unroll
			for (int i = 0; i < 4; i++)
				if (i < n) buf[slot[i]] = v[i];
		}
	};
	// every warp but the first for itself, the second for the first too
	auto fetch = [&](int h, uint32_t tag) {
		fetch_for((int)threadIdx.x, far, h, tag);
		if (wid == 1) fetch_for(lane, s_far[lane], h, tag);
	};
	if (wid == 0) s_far[lane] = far;
	// a warp's sum into s_red
	auto warp_pair = [&](const Dot &v, float2 *red) {
		Sum t = S::of(v);
#pragma unroll
		for (int o = 16; o > 0; o >>= 1) t = S::add(t, S::shfl(t, o));
		if (lane == 0) red[wid] = S::words(t);
	};
	// warp 0, after a block barrier: the CTA's sum to the group, and the group's
	auto send = [&](int v, ulonglong2 *row, uint32_t tag) {
		Sum t = S::of(s_red[v][lane & 15]);
#pragma unroll
		for (int o = 8; o > 0; o >>= 1) t = S::add(t, S::shfl(t, o));
		if (lane == 0) grid_put(row + rank, S::words(t), tag);
	};
	auto total = [&](const ulonglong2 *row, uint32_t tag) {
		Sum t = S::of(make_float2(0.f, 0.f));
		bool ok = true;
		constexpr int kRounds = 5;  // up to 160 CTAs
		const ulonglong2 *p[kRounds];
		float2 v[kRounds];
		int n = 0;
#pragma unroll
		for (int i = 0; i < kRounds; i++) {
			p[i] = row + lane + 32 * i;
			v[i] = make_float2(0.f, 0.f);
			n += lane + 32 * i < ctas;
		}
		if (n > 0) ok = grid_get(p, n, tag, v, A.st, limit);
#pragma unroll
		for (int i = 0; i < kRounds; i++)
			if (i < n) t = S::add(t, S::of(v[i]));
		__syncwarp();
#pragma unroll
		for (int o = 16; o > 0; o >>= 1) t = S::add(t, S::shfl(t, o));
		if (!ok) s_failed = 1;
		__syncwarp();
		return t;
	};
	// the first launch's numbers stay below the second's
	uint32_t tag = DBL ? 0x80000001u : 1u;  // of the current pairs
	publish(0, tag);
	warp_pair(acc, s_red[0]);
	if (PRE) warp_pair(accz, s_red[NV - 1]);
	__syncthreads();
	// warp 0 holds the solve's scalars
	Sum rho = S::of(make_float2(0.f, 0.f)), stop = rho;  // <r, z>; tol |r0|^2
	bool unsafe = false;
	int it = 0;
	if (wid != 0) {
		fetch(0, tag);
	} else {
		for (int v = 0; v < NV; v++) send(v, sums + (1 + v) * ctas, tag);
		const Sum nr0 = total(sums + ctas, tag);
		rho = PRE ? total(sums + NV * ctas, tag) : nr0;
		const double t = (double)A.a.tol * S::value(nr0);
		if constexpr (DBL) {
			stop = t;
		} else {
			stop.h = (float)t;
			stop.l = t < 3e38 ? (float)(t - (double)stop.h) : 0.f;
		}
		unsafe = !(S::safe(nr0) && S::safe(rho));
		if (lane == 0) s_active = s_failed ? kCgDone : unsafe ? kCgUnsafe : S::value(nr0) > 0.0 ? kCgOn : kCgDone;
	}
	__syncthreads();
	int active = s_active;
	float beta = 0.f;
	int h = 0;  // buffer of the current pairs
	while (active == kCgOn) {
		// d = z + beta d_old (own and neighbours) ; q = A d ; <z, q>
		const float2 *buf = s_pair + h * slots;
		acc = Dot();
#pragma unroll
		for (int u = 0; u < U; u++) {
			if ((int)threadIdx.x + u * kClusterBlock >= own) break;
			const float2 vu = buf[nud[u] & 0xFFFF], vl = buf[nlr[u] & 0xFFFF];
			const float2 vd = buf[nud[u] >> 16], vr = buf[nlr[u] >> 16];
			const float rk = PRE ? fm(minv[u], r[u]) : r[u];
			const float dk = fmaf(beta, d[u], rk);
			// a neighbour outside the hole reads zeros
			float lap = fm(-dk, sum[u]);
			lap = fmaf(su[u], fmaf(beta, vu.y, vu.x), lap);
			lap = fmaf(sl[u], fmaf(beta, vl.y, vl.x), lap);
			lap = fmaf(sc[u], fmaf(beta, vd.y, vd.x), lap);
			lap = fmaf(sc[u], fmaf(beta, vr.y, vr.x), lap);
			q[u] = fmaf(ls[u], dk, -fm(oml, lap));
			d[u] = dk;
			acc.add(rk, q[u]);
		}
		warp_pair(acc, s_red[0]);
		__syncthreads();
		if (wid == 0) {
			send(0, sums, tag);
			const Sum rq = total(sums, tag);
			const float alpha = S::quotient(rho, rq);
			unsafe = !DBL && !(S::safe(rq) && wide_safe(alpha));
			if (lane == 0) s_coef = alpha;
		}
		__syncthreads();
		const float alpha = s_coef;
		// r -= alpha q ; z = M r ; |r|^2 (and <r, z>) ; x += alpha d
		acc = Dot();
		accz = Dot();
#pragma unroll
		for (int u = 0; u < U; u++) {
			if ((int)threadIdx.x + u * kClusterBlock >= own) break;
			r[u] = fmaf(-alpha, q[u], r[u]);
			acc.add(r[u], r[u]);
			if (PRE) accz.add(r[u], fm(minv[u], r[u]));
		}
		h = 1 - h;
		tag++;
		publish(h, tag);
		warp_pair(acc, s_red[0]);
		if (PRE) warp_pair(accz, s_red[NV - 1]);
		__syncthreads();
		if (wid != 0) {
			fetch(h, tag);
		} else {
			for (int v = 0; v < NV; v++) send(v, sums + (1 + v) * ctas, tag);
			const Sum nrn = total(sums + ctas, tag);
			const Sum rhon = PRE ? total(sums + NV * ctas, tag) : nrn;
			const float bt = S::quotient(rhon, rho);
			// what underflows in |r|^2 does not matter below a threshold that is safe
			const bool done = (S::safe(nrn) || S::safe(stop)) && S::below(nrn, stop);
			if (lane == 0) {
				s_coef = bt;
				s_active = s_failed                                             ? kCgDone
				           : unsafe                                             ? kCgUnsafe
				           : done || it >= A.a.limit                            ? kCgDone
				           : DBL || (S::safe(nrn) && S::safe(rhon) && wide_safe(bt)) ? kCgOn
				                                                                : kCgUnsafe;
			}
			rho = rhon;
			it++;
		}
#pragma unroll
		for (int u = 0; u < U; u++) {
			if ((int)threadIdx.x + u * kClusterBlock >= own) break;
			x[u] = fmaf(alpha, d[u], x[u]);
		}
		// s_coef and s_active change only after the next block barrier, by
		// which every thread has read them
		__syncthreads();
		beta = s_coef;
		active = s_active;
	}
	if (rank == 0 && threadIdx.x == 0) {
		A.iters[ch] = it;
		if (!DBL) A.redo[ch] = active == kCgUnsafe;
	}
	if (s_failed) return;  // reported by the status word
	if (active == kCgUnsafe) return;
	// u = orig + delta on the hole (:89-104)
	double dacc = 0.0;
#pragma unroll
	for (int u = 0; u < U; u++) {
		const int l = threadIdx.x + u * kClusterBlock;
		if (l >= own) break;
		const int pix = A.hole[lo + l];
		const float o = A.orig[(size_t)C * pix + ch];
		const float v = o + x[u];
		const float prev = A.img[(size_t)C * pix + ch];
		const float dd = prev - v;
		dacc += (double)(dd * dd);
		A.img[(size_t)C * pix + ch] = v;
	}
	dacc = block_sum<kClusterBlock>(dacc, s_dbl);
	if (threadIdx.x == 0) A.diff[ch * ctas + rank] = dacc;
}

NLI_CHECK_READER(check_word_update)

static double read_total(nli_ctx *ctx, double *partials, int n, int *cg_iters_dev, int C, int nh = 0)
{
	launch_sum_partials(ctx->stream, partials, n, partials + n);
	char *h = static_cast<char *>(ctx->host_pinned);
	NLI_CUDA(cudaMemcpyAsync(h, partials + n, sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
	if (cg_iters_dev)
		NLI_CUDA(cudaMemcpyAsync(h + 64, cg_iters_dev, sizeof(int) * 4, cudaMemcpyDeviceToHost, ctx->stream));
	// timeouts of the waits of this iteration's kernels (PatchMatch's tensor
	// copies, CG grid barriers)
	NLI_CUDA(cudaMemcpyAsync(h + 128, &ctx->status->timeout, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
	NLI_CUDA(cudaStreamSynchronize(ctx->stream));
	if (*reinterpret_cast<const int *>(h + 128) != 0) {
		clear_timeout(ctx);
		NLI_REQUIRE(false, NLI_E_TIMEOUT, "a device-side wait timed out");
	}
	if (cg_iters_dev) {
		const int *it = reinterpret_cast<const int *>(h + 64);
		for (int c = 0; c < C; c++) {
			ctx->cg_iterations += it[c];
			ctx->cg_unknown_iterations += (int64_t)it[c] * nh;
		}
	}
	return *reinterpret_cast<double *>(h);
}

typedef void (*CgKernel)(PoissonArgs, int, const UnkC *, const float *, const float *, int *, const int32_t *,
                         const float *, float *, double *, int *);

template <bool PRE>
static CgKernel cg_kernel(bool single, int per)
{
	if (per == 2) return single ? k_poisson_cg_cta<PRE, 2> : k_poisson_cg_cluster<PRE, 2>;
	if (per == 5) return single ? k_poisson_cg_cta<PRE, 5> : k_poisson_cg_cluster<PRE, 5>;
	return single ? k_poisson_cg_cta<PRE, 8> : k_poisson_cg_cluster<PRE, 8>;
}

static CgKernel cg_kernel(bool pre, bool single, int per)
{
	return pre ? cg_kernel<true>(single, per) : cg_kernel<false>(single, per);
}

constexpr int kCgPerThread[] = {2, 5, 8};  // cg_per_thread's values

constexpr size_t kSmemBudget = 216 * 1024;
static_assert(2 * sizeof(float2) * (3 * kClusterMaxChunk + 3) <= kSmemBudget, "every chunk fits a CTA");

// Solver layout of a system of nh unknowns per channel: *ncta CTAs of
// *chunk unknowns each (one CTA with block barriers when *ncta is 1, a
// cluster when it is more), or *ncta = 0 for the cooperative grid CG.
static void cg_layout(nli_ctx *ctx, int nh, int *ncta, int *chunk)
{
	if (ctx->cg_cluster_max < 0) {
		// largest cluster the device runs with the biggest shared-memory footprint
		int maxc = 0;
		bool ok = true;
		for (int pre = 0; pre < 2; pre++)
			for (int per : kCgPerThread) {
				const CgKernel cluster = cg_kernel(pre, false, per), cta = cg_kernel(pre, true, per);
				ok &= cudaFuncSetAttribute(cluster, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == 0;
				ok &= cudaFuncSetAttribute(cluster, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemBudget) == 0;
				ok &= cudaFuncSetAttribute(cta, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemBudget) == 0;
			}
		if (ok) {
			cudaLaunchConfig_t qc = {};
			qc.gridDim = dim3(kClusterMax);
			qc.blockDim = dim3(kClusterBlock);
			qc.dynamicSmemBytes = kSmemBudget;
			if (cudaOccupancyMaxPotentialClusterSize(&maxc, cg_kernel(true, false, kClusterPerThread), &qc) !=
			    cudaSuccess)
				maxc = 0;
		}
		cudaGetLastError();
		ctx->cg_cluster_max = std::min(maxc, kClusterMax);
	}
	*ncta = *chunk = 0;
	if (ctx->cg_cluster_max >= 1) {
		const int per = std::max(1, ctx->tune_cg_unknowns_per_cta);
		*ncta = std::max(1, std::min(std::min(ctx->cg_cluster_max, ctx->tune_cg_cluster_cap), (nh + per - 1) / per));
		*chunk = (nh + *ncta - 1) / *ncta;
		// (a 16-bit code names a neighbour, and the last one means none)
		if (*chunk > kClusterMaxChunk || nh > kNoNb) *ncta = *chunk = 0;
		// small systems: one CTA, block barriers only (NLI_TUNE_CG_SINGLE_MAX)
		if (nh <= std::min(ctx->tune_cg_single_max, kClusterMaxChunk)) {
			*ncta = 1;
			*chunk = nh;
		}
	}
}

// Coefficients (gather), the compact system and its right-hand side b and
// start x0 = image - orig (patch_non_local_poisson.cpp:36-82).  Chooses the
// solver layout: `chunk` / `ncta` > 0 for the cluster CG.
struct PoissonSystem {
	PoissonArgs pa;
	CoefOut co;
	const float4 *pad;  // the image as padded pixels
	Unknown *unk = nullptr;  // grid layouts
	UnkC *unkc = nullptr;    // cluster layouts
	float *b, *x;
	int chunk = 0, ncta = 0;
};

static PoissonSystem poisson_system(nli_ctx *ctx, const UpdArgs &u, const nli_update_params &up, const float *image,
                                    const float *orig, const uint8_t *dom, const uint8_t *ext, const int2 *nnf,
                                    const float *conf, const int32_t *hole, int nh)
{
	cudaStream_t s = ctx->stream;
	const int W = u.W, H = u.H, C = u.C;
	const size_t n = (size_t)W * H;
	PoissonSystem P;
	float4 *pad = ctx->buf<float4>("poi.pad", (size_t)(W + 1) * (H + 1));
	launch_pad4(s, image, W, H, C, pad);
	P.pad = pad;
	int32_t *index = ctx->buf<int32_t>("upd.hole_index", n);
	P.co.S = ctx->buf<float>("poi.S", n);
	P.co.U = ctx->buf<float>("poi.U", n * C);
	P.co.GX = ctx->buf<float>("poi.GX", n * C);
	P.co.GY = ctx->buf<float>("poi.GY", n * C);
	with_channels(C, [&](auto c) {
		constexpr int CC = decltype(c)::value;
		ProfScope ps(ctx, "poisson_coef");
		if (u.px % 2 == 1 && u.py % 2 == 1) {
			const long long threads = 3LL * nh * 8;
			launch_early(s, (int)((threads + 255) / 256), 256, 0, k_poisson_coef8<CC>, u, hole, nh, dom, ext, nnf, conf, pad, P.co,
			                                                                 index);
		} else {
			// even patch sides: the window of gather_coef is one wider than the patch
			launch_early(s, (nh + 127) / 128, 128, 0, k_poisson_coef<CC>, u, hole, nh, dom, ext, nnf, conf, pad, P.co, index);
		}
		NLI_CHECK_LAUNCH();
	});
	PoissonArgs &pa = P.pa;
	pa.W = W;
	pa.H = H;
	pa.C = C;
	pa.nh = nh;
	for (int c = 0; c < 4; c++) pa.lambda[c] = up.lambda;
	if (up.method == NLI_UPDATE_DEPTH) pa.lambda[3] = up.lambda_d;
	pa.tol = up.cg_tol;
	pa.limit = up.cg_iters;
	P.b = ctx->buf<float>("poi.b", (size_t)nh * C);
	P.x = ctx->buf<float>("poi.x", (size_t)nh * C);

	cg_layout(ctx, nh, &P.ncta, &P.chunk);
	if (P.ncta > 0)
		P.unkc = ctx->buf<UnkC>("poi.unkc", nh);
	else
		P.unk = ctx->buf<Unknown>("poi.unk", nh);
	{
		ProfScope ps(ctx, "poisson_setup");
		launch_early(s, (nh + 255) / 256, 256, 0, k_poisson_setup, pa, P.chunk, hole, dom, index, P.co, image, orig, P.unk,
		                                                  P.unkc, P.b, P.x);
		NLI_CHECK_LAUNCH();
	}
	return P;
}

// Layout of a system that is too large for a cluster: `groups` channels at a
// time on `ctas` CTAs each (k_poisson_cg_wide; as many channels at once as the
// SMs can hold, since an iteration costs two exchanges whatever its size), or
// groups = 0 for k_poisson_cg, which keeps its vectors in memory: more unknowns
// than the SMs hold, or rows too wide for a neighbour's distance.
struct GridLayout {
	int groups, ctas, chunk;
	int parts;  // partial sums of (du)^2
};

typedef void (*WideKernel)(GridCgArgs);

// two buffers of pairs and a word per unknown
static size_t wide_smem_bytes(int chunk) { return cg_smem_bytes(chunk) + sizeof(uint32_t) * (size_t)chunk; }
static_assert(2 * sizeof(float2) * (3 * kClusterMaxChunk + 3) + 4 * kClusterMaxChunk <= kSmemBudget, "every chunk fits");

template <bool DBL>
static WideKernel wide_kernel(bool pre, int chunk)
{
	if (chunk <= 5 * kClusterBlock) return pre ? k_poisson_cg_wide<true, 5, DBL> : k_poisson_cg_wide<false, 5, DBL>;
	return pre ? k_poisson_cg_wide<true, kClusterPerThread, DBL> : k_poisson_cg_wide<false, kClusterPerThread, DBL>;
}

static WideKernel wide_kernel(bool pre, int chunk, bool dbl)
{
	return dbl ? wide_kernel<true>(pre, chunk) : wide_kernel<false>(pre, chunk);
}

static GridLayout grid_layout(nli_ctx *ctx, int nh, int C, int W)
{
	GridLayout g = {0, 0, 0, 0};
	const bool pre = ctx->tune_cg_precond != 0;
	if (W <= 0xFFFF)
		for (int groups = C; groups >= 1 && g.groups == 0; groups--) {
			const int ctas = std::min({ctx->num_sms / groups, (nh + kClusterBlock - 1) / kClusterBlock, 160});
			const int chunk = ctas > 0 ? (nh + ctas - 1) / ctas : nh;
			if (chunk <= kClusterMaxChunk) g = {groups, ctas, chunk, C * ctas};
		}
	if (g.groups > 0) {
		static std::atomic<uint32_t> raised{0};  // one bit per device
		const uint32_t bit = 1u << (ctx->device & 31);
		if (!(raised.load(std::memory_order_acquire) & bit)) {
			for (int pr = 0; pr < 2; pr++)
				for (int c : {1, kClusterMaxChunk})
					for (int dbl = 0; dbl < 2; dbl++)
						NLI_CUDA(cudaFuncSetAttribute(wide_kernel(pr, c, dbl), cudaFuncAttributeMaxDynamicSharedMemorySize,
						                              (int)kSmemBudget));
			raised.fetch_or(bit, std::memory_order_release);
		}
		return g;
	}
	int per_sm = 0;
	const void *kern = pre ? (const void *)k_poisson_cg<true> : (const void *)k_poisson_cg<false>;
	NLI_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kCgBlock, 0));
	const int max_blocks = per_sm * ctx->num_sms;
	NLI_REQUIRE(max_blocks > 0, NLI_E_CUDA, "conjugate gradient kernel cannot be made resident");
	const int grid = (nh + kCgBlock - 1) / kCgBlock;
	g.ctas = g.parts = std::min(std::max(grid, 1), std::min(max_blocks, ctx->num_sms));
	return g;
}

// A cooperative launch through the launch attribute, which stream capture
// takes.
static void launch_cooperative(nli_ctx *ctx, const void *kern, int grid, int block, size_t smem, void **args)
{
	cudaLaunchConfig_t cfg = {};
	cfg.gridDim = dim3(grid);
	cfg.blockDim = dim3(block);
	cfg.dynamicSmemBytes = smem;
	cfg.stream = ctx->stream;
	cudaLaunchAttribute attr[1];
	attr[0].id = cudaLaunchAttributeCooperative;
	attr[0].val.cooperative = 1;
	cfg.attrs = attr;
	cfg.numAttrs = 1;
	NLI_CUDA(cudaLaunchKernelExC(&cfg, kern, args));
	nli_count_launch_internal();
}

// k_poisson_cg_wide for system P.  active (may be null): a device flag; 0
// makes every block leave at once.
static void launch_wide_cg(nli_ctx *ctx, const PoissonSystem &P, const GridLayout &g, int *iters, const int32_t *hole,
                           const float *orig, float *img, double *diff_part, const int *active)
{
	const bool pre = ctx->tune_cg_precond != 0;
	const int nh = P.pa.nh, C = P.pa.C, rows = pre ? 3 : 2;  // sums per group and CTA
	const size_t npairs = 2 * (size_t)g.groups * nh, nsums = (size_t)g.groups * rows * g.ctas;
	ulonglong2 *words = ctx->buf<ulonglong2>("poi.words", npairs + nsums);
	int *redo = ctx->buf<int>("poi.redo", 4);
	GridCgArgs A;
	A.a = P.pa;
	A.chunk = g.chunk;
	A.ctas = g.ctas;
	A.unk = P.unk;
	A.b = P.b;
	A.x0 = P.x;
	A.pairs = words;
	A.sums = words + npairs;
	A.st = ctx->status;
	A.iters = iters;
	A.redo = redo;
	A.hole = hole;
	A.orig = orig;
	A.img = img;
	A.diff = diff_part;
	A.active = active;
	ProfScope ps(ctx, "poisson_cg");
	for (int c = 0; c < C; c += g.groups) {
		A.ch0 = c;
		void *args[] = {&A};
		NLI_CUDA(cudaMemsetAsync(words, 0, sizeof(ulonglong2) * (npairs + nsums), ctx->stream));
		for (int dbl = 0; dbl < 2; dbl++)
			launch_cooperative(ctx, (const void *)wide_kernel(pre, g.chunk, dbl), std::min(g.groups, C - c) * g.ctas,
			                   kClusterBlock, wide_smem_bytes(g.chunk), args);
	}
}

struct GridCgBufs {
	float *r, *d, *q, *z;  // nh * C each (z only when preconditioned)
	double *part;          // grid * 16
};

// The cooperative grid CG of system P on `grid` blocks.  active (may be
// null): a device flag; 0 makes every block leave at once.
static void launch_grid_cg(nli_ctx *ctx, const PoissonSystem &P, int grid, const GridCgBufs &g, int *iters,
                           const int32_t *hole, const float *orig, float *img, double *diff_part, const int *active)
{
	cudaStream_t s = ctx->stream;
	const bool pre = ctx->tune_cg_precond != 0;
	const void *kern = pre ? (const void *)k_poisson_cg<true> : (const void *)k_poisson_cg<false>;
	// the grid barrier's counters (the timeout word is left for the
	// iteration's readback)
	NLI_CUDA(cudaMemsetAsync(ctx->status, 0, offsetof(DevStatus, timeout), s));
	DevStatus *st = ctx->status;
	PoissonArgs pa = P.pa;
	const Unknown *unk = P.unk;
	const float *b = P.b;
	float *x = P.x;
	float *r = g.r, *d = g.d, *q = g.q, *z = g.z;
	double *part = g.part;
	void *args[] = {&pa,   &unk, &b,     &x,    (void *)&r, &d,         &q,         &z,
	                &part, &st,  &iters, (void *)&hole, &orig, &img, &diff_part, (void *)&active};
	ProfScope ps(ctx, "poisson_cg");
	launch_cooperative(ctx, kern, grid, kCgBlock, 0, args);
}

// Solves the system from x0 (the CG of :387-477) and writes u = orig + x on
// the hole into img, with per-block partial sums of (u_old - u_new)^2 in
// "poi.diff" (returns their count).
static int poisson_solve(nli_ctx *ctx, PoissonSystem &P, const int32_t *hole, const float *orig, float *img)
{
	cudaStream_t s = ctx->stream;
	const int nh = P.pa.nh, C = P.pa.C;
	int *iters = ctx->buf<int>("poi.iters", 4);
	if (P.ncta > 0) {
		const bool pre = ctx->tune_cg_precond != 0;
		const size_t smem = cg_smem_bytes(P.chunk);
		const CgKernel kern = cg_kernel(pre, P.ncta == 1, cg_per_thread(P.chunk));
		double *diff_part = ctx->buf<double>("poi.diff", (size_t)C * P.ncta + 1);
		if (P.ncta == 1) {
			// one CTA per channel: no cluster
			ProfScope ps(ctx, "poisson_cg");
			kern<<<C, kClusterBlock, smem, s>>>(P.pa, P.chunk, P.unkc, P.b, P.x, iters, hole, orig, img, diff_part,
			                                    &ctx->status->timeout);
			NLI_CHECK_LAUNCH();
			return C;
		}
		cudaLaunchConfig_t cfg = {};
		cfg.gridDim = dim3(C * P.ncta);
		cfg.blockDim = dim3(kClusterBlock);
		cfg.dynamicSmemBytes = smem;
		cfg.stream = s;
		cudaLaunchAttribute attr[1];
		attr[0].id = cudaLaunchAttributeClusterDimension;
		attr[0].val.clusterDim.x = P.ncta;
		attr[0].val.clusterDim.y = 1;
		attr[0].val.clusterDim.z = 1;
		cfg.attrs = attr;
		cfg.numAttrs = 1;
		ProfScope ps(ctx, "poisson_cg");
		NLI_CUDA(cudaLaunchKernelEx(&cfg, kern, P.pa, P.chunk, (const UnkC *)P.unkc, (const float *)P.b,
		                            (const float *)P.x, iters, hole, orig, img, diff_part, &ctx->status->timeout));
		nli_count_launch_internal();
		return C * P.ncta;
	}
	const GridLayout gl = grid_layout(ctx, nh, C, P.pa.W);
	if (gl.groups > 0) {
		double *diff_part = ctx->buf<double>("poi.diff", gl.parts + 1);
		launch_wide_cg(ctx, P, gl, iters, hole, orig, img, diff_part, nullptr);
		return gl.parts;
	}
	const int grid = gl.ctas;
	double *part = ctx->buf<double>("poi.part", (size_t)grid * 16);
	double *diff_part = ctx->buf<double>("poi.diff", grid + 1);
	GridCgBufs g;
	g.r = ctx->buf<float>("poi.r", (size_t)nh * C);
	g.d = ctx->buf<float>("poi.d", (size_t)nh * C);
	g.q = ctx->buf<float>("poi.q", (size_t)nh * C);
	g.z = ctx->tune_cg_precond ? ctx->buf<float>("poi.z", (size_t)nh * C) : nullptr;
	g.part = part;
	launch_grid_cg(ctx, P, grid, g, iters, hole, orig, img, diff_part, nullptr);
	return grid;
}

static void poisson_run(nli_ctx *ctx, const UpdArgs &u, const nli_update_params &up, float *image, const float *orig,
                        const uint8_t *dom, const uint8_t *ext, const int2 *nnf, const float *conf,
                        const int32_t *hole, int nh, int *n_partials)
{
	PoissonSystem P = poisson_system(ctx, u, up, image, orig, dom, ext, nnf, conf, hole, nh);
	*n_partials = poisson_solve(ctx, P, hole, orig, image);
}

double update_run(nli_ctx *ctx, const nli_update_params &up, float *image, const float *orig, const uint8_t *dom,
                  const uint8_t *ext, const int32_t *nnf_i, const float *conf, int W, int H, int C,
                  const int32_t *hole, int nh, bool read_back, const double **total_dev, const int **cg_iters_dev)
{
	NLI_REQUIRE(up.method >= 0 && up.method <= 3, NLI_E_UNSUPPORTED, "unknown update method");
	if (up.method == NLI_UPDATE_DEPTH) NLI_REQUIRE(C == 4, NLI_E_CHANNELS, "Separate: Channels do not match.");
	UpdArgs u;
	fill_upd_args(u, up, W, H, C);
	cudaStream_t s = ctx->stream;
	const int2 *nnf = reinterpret_cast<const int2 *>(nnf_i);
	if (!hole) {
		int32_t *l = ctx->buf<int32_t>("upd.hole", (size_t)W * H);
		nh = compact_mask(ctx, dom, W, H, l, "upd");
		hole = l;
	}
	if (nh <= 0) return 0.0;
	if (up.method == NLI_UPDATE_POISSON || up.method == NLI_UPDATE_DEPTH) {
		int np = 0;
		poisson_run(ctx, u, up, image, orig, dom, ext, nnf, conf, hole, nh, &np);
		double *diff_part = ctx->buf<double>("poi.diff", np + 1);
		if (!read_back) {
			launch_sum_partials(s, diff_part, np, diff_part + np);
			if (total_dev) *total_dev = diff_part + np;
			if (cg_iters_dev) *cg_iters_dev = ctx->buf<int>("poi.iters", 4);
			return 0.0;
		}
		return read_total(ctx, diff_part, np, ctx->buf<int>("poi.iters", 4), C, nh);
	}
	float *newval = ctx->buf<float>("upd.newval", (size_t)nh * C);
	int grid;
	double *partials;
	if (up.method == NLI_UPDATE_MEANS) {
		grid = (int)(((long long)nh * C + 255) / 256);
		partials = ctx->buf<double>("upd.partials", grid + 1);
		ProfScope ps(ctx, "nlmeans");
		launch_early(s, grid, 256, 0, k_nlmeans, u, image, hole, nh, dom, nnf, conf, newval, partials);
	} else {
		grid = (nh + kMedWarps - 1) / kMedWarps;
		partials = ctx->buf<double>("upd.partials", grid + 1);
		ProfScope ps(ctx, "nlmedians");
		if (med_window(u) <= 32 * kMedSmall)
			launch_early(s, grid, 32 * kMedWarps, 0, k_nlmedians<kMedSmall>, u, image, hole, nh, dom, nnf, conf, newval,
			                                                       partials);
		else
			launch_early(s, grid, 32 * kMedWarps, 0, k_nlmedians<kMedLarge>, u, image, hole, nh, dom, nnf, conf, newval,
			                                                       partials);
	}
	NLI_CHECK_LAUNCH();
	launch_early(s, (nh * C + 255) / 256, 256, 0, k_scatter_values, hole, nh, C, newval, image);
	NLI_CHECK_LAUNCH();
	if (!read_back) {
		launch_sum_partials(s, partials, grid, partials + grid);
		if (total_dev) *total_dev = partials + grid;
		if (cg_iters_dev) *cg_iters_dev = nullptr;
		return 0.0;
	}
	return read_total(ctx, partials, grid, nullptr, C);
}

// ======================================================= batched updates
// The update step of up to kBatchMax images in one launch per kernel (the
// lockstep batch driver, process.cu).  Each image keeps its own sizes,
// method, lambda and CG tolerance; the patch and its weights are shared.
// Every per-pixel / per-unknown value comes from the same device functions
// as the one-image kernels, and every reduction keeps the one-image
// partition (blocks of one image never straddle another image; each CG
// system has the same CTA layout), so each image's result and its sum of
// (u_old - u_new)^2 equal those of its one-image update bit for bit.
// Images whose active flag is 0 are skipped.  The per-image arguments
// travel in kernel parameter space (__grid_constant__ tables).
struct BTask {
	int img_index;  // index of the image's active flag
	int W, H, nh;
	float *img;
	const float *orig;
	const uint8_t *dom, *ext;
	const int2 *nnf;
	const float *conf;
	const int32_t *hole;
	float *newval;      // NL-means / NL-medians: new values of the hole
	double *partials;   // NL-means / NL-medians: per-block sums
	int32_t *hidx;      // NL-Poisson: unknown index per pixel
	float4 *pad;        // NL-Poisson: the image as padded pixels
	CoefOut co;
	Unknown *unk;
	UnkC *unkc;
	float *b, *x;
	PoissonArgs pa;
	int chunk, ncta;    // CG layout (ncta 0: grid CG)
	int *iters;
	double *diff;       // CG: partial sums of (du)^2
	int nparts;         // partial sums behind `total`
	double *total;      // this step's sum of (du)^2
};

struct BArgs {
	int n;
	const int *active;
	int blk[kBatchMax + 1];  // block prefix of the launch
	BTask t[kBatchMax];
};

__device__ __forceinline__ bool btask_on(const BArgs &B, int t) { return !B.active || B.active[B.t[t].img_index]; }

// The task whose block range [blk[t], blk[t + 1]) holds block b.
__device__ __forceinline__ int task_of_block(const BArgs &B, int b)
{
	int lo = 0, hi = B.n;
	while (hi - lo > 1) {
		const int mid = (lo + hi) >> 1;
		if (B.blk[mid] <= b)
			lo = mid;
		else
			hi = mid;
	}
	return lo;
}

__global__ void __launch_bounds__(256) k_nlmeans_batch(UpdArgs u, const __grid_constant__ BArgs B, int C)
{
	__shared__ double red[8];
	const int t = task_of_block(B, blockIdx.x);
	if (!btask_on(B, t)) return;
	const BTask &T = B.t[t];
	const int bl = blockIdx.x - B.blk[t];
	const int i = bl * 256 + (int)threadIdx.x;
	const int k = i / C, c = i - k * C;
	float sq = 0.f;
	if (k < T.nh) sq = nlmeans_value(u, T.W, T.H, C, c, T.img, T.hole[k], T.dom, T.nnf, T.conf, T.newval[i]);
	const double acc = block_sum<256>((double)sq, red);
	if (threadIdx.x == 0) T.partials[bl] = acc;
}

template <int NB>
__global__ void __launch_bounds__(32 * kMedWarps) k_nlmedians_batch(UpdArgs u, const __grid_constant__ BArgs B, int C)
{
	__shared__ __align__(16) MedSmem<NB> sm[kMedWarps];
	__shared__ double red[kMedWarps];
	const int t = task_of_block(B, blockIdx.x);
	if (!btask_on(B, t)) return;
	const BTask &T = B.t[t];
	const int bl = blockIdx.x - B.blk[t];
	const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
	const int i = bl * kMedWarps + wid;
	double acc = 0.0;
	if (i < T.nh)
		acc = nlmedians_pixel<NB>(u, T.W, T.H, C, T.img, T.hole[i], T.dom, T.nnf, T.conf, T.newval + (size_t)C * i,
		                      sm[wid]);
	if (lane == 0) red[wid] = acc;
	__syncthreads();
	if (threadIdx.x == 0) {
		double tt = 0.0;
		for (int w = 0; w < kMedWarps; w++) tt += red[w];
		T.partials[bl] = tt;
	}
}

// New values into the image (k_scatter_values per image).
__global__ void k_scatter_batch(const __grid_constant__ BArgs B, int C)
{
	const int t = blockIdx.y;
	if (!btask_on(B, t)) return;
	const BTask &T = B.t[t];
	for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < T.nh * C; i += gridDim.x * blockDim.x) {
		const int k = i / C, c = i % C;
		T.img[(size_t)C * T.hole[k] + c] = T.newval[i];
	}
}

// The image's sum of (du)^2 from its partial sums (k_sum_partials per
// image: one 1024-thread block each, the same order).  which 0: the
// NL-means / NL-medians block sums, 1: the CG partial sums.
__global__ void __launch_bounds__(1024) k_total_batch(const __grid_constant__ BArgs B, int which)
{
	__shared__ double sm[32];
	const int t = blockIdx.x;
	if (!btask_on(B, t)) return;
	const BTask &T = B.t[t];
	const double *part = which ? T.diff : T.partials;
	double v = 0.0;
	for (int i = threadIdx.x; i < T.nparts; i += blockDim.x) v += part[i];
	v = block_sum<1024>(v, sm);
	if (threadIdx.x == 0) *T.total = v;
}

__global__ void k_upd_pad_batch(const __grid_constant__ BArgs B, int C)
{
	const int t = blockIdx.y;
	if (!btask_on(B, t)) return;
	const BTask &T = B.t[t];
	pad4_span(T.img, T.W, T.H, C, T.pad, blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x);
}

template <int C>
__global__ void __launch_bounds__(256) k_coef8_batch(UpdArgs u, const __grid_constant__ BArgs B)
{
	const int t = task_of_block(B, blockIdx.x);
	if (!btask_on(B, t)) return;
	const BTask &T = B.t[t];
	const int item = (((int)blockIdx.x - B.blk[t]) * 256 + (int)threadIdx.x) >> 3;
	coef8_item<C>(u, T.W, T.H, item, threadIdx.x & 7, T.hole, T.nh, T.dom, T.ext, T.nnf, T.conf, T.pad, T.co, T.hidx);
}

template <int C>
__global__ void __launch_bounds__(128) k_coef_batch(UpdArgs u, const __grid_constant__ BArgs B)
{
	const int t = task_of_block(B, blockIdx.x);
	if (!btask_on(B, t)) return;
	const BTask &T = B.t[t];
	const int i = ((int)blockIdx.x - B.blk[t]) * 128 + (int)threadIdx.x;
	if (i >= T.nh) return;
	coef_hole_pixel<C>(u, T.W, T.H, i, T.hole, T.dom, T.ext, T.nnf, T.conf, T.pad, T.co, T.hidx);
}

__global__ void k_setup_batch(const __grid_constant__ BArgs B)
{
	const int t = task_of_block(B, blockIdx.x);
	if (!btask_on(B, t)) return;
	const BTask &T = B.t[t];
	const int k = ((int)blockIdx.x - B.blk[t]) * 256 + (int)threadIdx.x;
	if (k >= T.nh) return;
	poisson_setup_unknown(T.pa, T.chunk, k, T.hole, T.dom, T.hidx, T.co, T.img, T.orig, T.unk, T.unkc, T.b, T.x);
}

// CG systems of one layout class (the same CTAs per system): system g of
// the launch is channel g % C of task g / C.
struct CgTask {
	int img_index;
	PoissonArgs a;
	int chunk;
	const UnkC *unk;
	const float *b, *x0;
	int *iters;
	const int32_t *hole;
	const float *orig;
	float *img;
	double *diff;
};

struct CgArgs {
	int n, C, ncta;
	const int *active;
	int *timeout;
	CgTask t[kBatchMax];
};

template <bool PRE, bool SINGLE, int U>
__global__ void __launch_bounds__(kClusterBlock, 1) k_poisson_cg_batch(const __grid_constant__ CgArgs B)
{
	const int ncta = SINGLE ? 1 : B.ncta;
	const int g = (int)blockIdx.x / ncta;
	const int t = g / B.C, group = g - t * B.C;
	const CgTask &T = B.t[t];
	// a stopped image: every CTA of its clusters leaves before any barrier
	if (B.active && !B.active[T.img_index]) return;
	cg_team_solve<PRE, SINGLE, U>(T.a, T.chunk, T.unk, T.b, T.x0, T.iters, T.hole, T.orig, T.img, T.diff, group,
	                              B.timeout);
}

template <bool PRE>
static void (*cg_batch_kernel(bool single, int per))(CgArgs)
{
	if (per == 2) return single ? k_poisson_cg_batch<PRE, true, 2> : k_poisson_cg_batch<PRE, false, 2>;
	if (per == 5) return single ? k_poisson_cg_batch<PRE, true, 5> : k_poisson_cg_batch<PRE, false, 5>;
	return single ? k_poisson_cg_batch<PRE, true, 8> : k_poisson_cg_batch<PRE, false, 8>;
}

static void (*cg_batch_kernel(bool pre, bool single, int per))(CgArgs)
{
	return pre ? cg_batch_kernel<true>(single, per) : cg_batch_kernel<false>(single, per);
}

static std::string lk_name(int i, const char *what) { return "lk." + std::to_string(i) + "." + what; }

static int div_up(long long a, int b) { return (int)((a + b - 1) / b); }

// Elementwise launch over n images: blockIdx.y = image, grid-stride in x.
static dim3 per_image_grid(long long maxcount, int n, int block = 256)
{
	return dim3((unsigned)std::max(1, std::min(div_up(maxcount, block), 1024)), (unsigned)n);
}

void update_batch_run(nli_ctx *ctx, const nli_update_params *ups, int C, int n, const UpdBatchItem *items,
                      const int *active)
{
	NLI_REQUIRE(n >= 1 && n <= kBatchMax, NLI_E_INVALID, "batched updates take 1 to 64 images");
	cudaStream_t s = ctx->stream;
	UpdArgs u;
	fill_upd_args(u, ups[0], 0, 0, C);
	for (int i = 1; i < n; i++)
		NLI_REQUIRE(ups[i].patch_x == ups[0].patch_x && ups[i].patch_y == ups[0].patch_y &&
		                ups[i].sigma == ups[0].sigma,
		            NLI_E_INVALID, "batched updates share the patch and its sigma");
	BArgs M, D, P;  // NL-means, NL-medians, NL-Poisson / NL-depth images
	std::memset(&M, 0, sizeof(M));
	std::memset(&D, 0, sizeof(D));
	std::memset(&P, 0, sizeof(P));
	M.active = D.active = P.active = active;
	long long maxnh = 0, maxpad = 0;
	for (int i = 0; i < n; i++) {
		const UpdBatchItem &it = items[i];
		const nli_update_params &up = ups[i];
		NLI_REQUIRE(up.method >= 0 && up.method <= 3, NLI_E_UNSUPPORTED, "unknown update method");
		if (up.method == NLI_UPDATE_DEPTH) NLI_REQUIRE(C == 4, NLI_E_CHANNELS, "Separate: Channels do not match.");
		BArgs &B = (up.method == NLI_UPDATE_MEANS) ? M : (up.method == NLI_UPDATE_MEDIANS) ? D : P;
		BTask &T = B.t[B.n++];
		T.img_index = it.flag;
		T.W = it.W;
		T.H = it.H;
		T.nh = it.nh;
		T.img = it.img;
		T.orig = it.orig;
		T.dom = it.dom;
		T.ext = it.ext;
		T.nnf = reinterpret_cast<const int2 *>(it.nnf);
		T.conf = it.conf;
		T.hole = it.hole;
		T.total = it.total;
		T.iters = it.cg_iters;
		maxnh = std::max<long long>(maxnh, it.nh);
		const size_t np = (size_t)it.W * it.H;
		const size_t nh = (size_t)std::max(it.nh, 1);
		if (&B != &P) {
			T.nparts = (&B == &M) ? div_up((long long)it.nh * C, 256) : div_up(it.nh, kMedWarps);
			T.newval = ctx->buf<float>(lk_name(it.flag, "newval"), nh * C);
			T.partials = ctx->buf<double>(lk_name(it.flag, "partials"), (size_t)std::max(T.nparts, 1));
			continue;
		}
		PoissonArgs &pa = T.pa;
		pa.W = it.W;
		pa.H = it.H;
		pa.C = C;
		pa.nh = it.nh;
		for (int c = 0; c < 4; c++) pa.lambda[c] = up.lambda;
		if (up.method == NLI_UPDATE_DEPTH) pa.lambda[3] = up.lambda_d;
		pa.tol = up.cg_tol;
		pa.limit = up.cg_iters;
		T.hidx = ctx->buf<int32_t>(lk_name(it.flag, "hidx"), np);
		T.pad = ctx->buf<float4>(lk_name(it.flag, "pad"), (size_t)(it.W + 1) * (it.H + 1));
		maxpad = std::max(maxpad, (long long)(it.W + 1) * (it.H + 1));
		T.co.S = ctx->buf<float>(lk_name(it.flag, "S"), np);
		T.co.U = ctx->buf<float>(lk_name(it.flag, "U"), np * C);
		T.co.GX = ctx->buf<float>(lk_name(it.flag, "GX"), np * C);
		T.co.GY = ctx->buf<float>(lk_name(it.flag, "GY"), np * C);
		T.b = ctx->buf<float>(lk_name(it.flag, "b"), nh * C);
		T.x = ctx->buf<float>(lk_name(it.flag, "x"), nh * C);
		cg_layout(ctx, it.nh, &T.ncta, &T.chunk);
		if (it.nh == 0) {
			T.nparts = 0;  // nothing to solve: the step's sum is 0
		} else if (T.ncta > 0) {
			T.unkc = ctx->buf<UnkC>(lk_name(it.flag, "unkc"), nh);
			T.nparts = C * T.ncta;
		} else {
			T.unk = ctx->buf<Unknown>(lk_name(it.flag, "unk"), nh);
			T.nparts = grid_layout(ctx, it.nh, C, it.W).parts;
		}
		T.diff = ctx->buf<double>(lk_name(it.flag, "diff"), (size_t)T.nparts + 1);
	}
	const int blk = 256;
	// ---- NL-means
	if (M.n > 0) {
		for (int t = 0; t < M.n; t++) M.blk[t + 1] = M.blk[t] + M.t[t].nparts;
		if (M.blk[M.n] > 0) {
			ProfScope ps(ctx, "nlmeans");
			k_nlmeans_batch<<<M.blk[M.n], 256, 0, s>>>(u, M, C);
			NLI_CHECK_LAUNCH();
		}
		k_scatter_batch<<<per_image_grid(maxnh * C, M.n), blk, 0, s>>>(M, C);
		NLI_CHECK_LAUNCH();
		k_total_batch<<<M.n, 1024, 0, s>>>(M, 0);
		NLI_CHECK_LAUNCH();
	}
	// ---- NL-medians
	if (D.n > 0) {
		for (int t = 0; t < D.n; t++) D.blk[t + 1] = D.blk[t] + div_up(D.t[t].nh, kMedWarps);
		if (D.blk[D.n] > 0) {
			ProfScope ps(ctx, "nlmedians");
			if (med_window(u) <= 32 * kMedSmall)
				k_nlmedians_batch<kMedSmall><<<D.blk[D.n], 32 * kMedWarps, 0, s>>>(u, D, C);
			else
				k_nlmedians_batch<kMedLarge><<<D.blk[D.n], 32 * kMedWarps, 0, s>>>(u, D, C);
			NLI_CHECK_LAUNCH();
		}
		k_scatter_batch<<<per_image_grid(maxnh * C, D.n), blk, 0, s>>>(D, C);
		NLI_CHECK_LAUNCH();
		k_total_batch<<<D.n, 1024, 0, s>>>(D, 0);
		NLI_CHECK_LAUNCH();
	}
	if (P.n == 0) return;
	// ---- NL-Poisson / NL-depth: system set-up for every image
	k_upd_pad_batch<<<per_image_grid(maxpad, P.n), blk, 0, s>>>(P, C);
	NLI_CHECK_LAUNCH();
	with_channels(C, [&](auto c) {
		constexpr int CC = decltype(c)::value;
		ProfScope ps(ctx, "poisson_coef");
		if (u.px % 2 == 1 && u.py % 2 == 1) {
			for (int t = 0; t < P.n; t++) P.blk[t + 1] = P.blk[t] + div_up(3LL * P.t[t].nh * 8, 256);
			if (P.blk[P.n] > 0) k_coef8_batch<CC><<<P.blk[P.n], 256, 0, s>>>(u, P);
		} else {
			for (int t = 0; t < P.n; t++) P.blk[t + 1] = P.blk[t] + div_up(P.t[t].nh, 128);
			if (P.blk[P.n] > 0) k_coef_batch<CC><<<P.blk[P.n], 128, 0, s>>>(u, P);
		}
		if (P.blk[P.n] > 0) NLI_CHECK_LAUNCH();
	});
	{
		ProfScope ps(ctx, "poisson_setup");
		for (int t = 0; t < P.n; t++) P.blk[t + 1] = P.blk[t] + div_up(P.t[t].nh, 256);
		if (P.blk[P.n] > 0) {
			k_setup_batch<<<P.blk[P.n], 256, 0, s>>>(P);
			NLI_CHECK_LAUNCH();
		}
	}
	// ---- the solves, one launch per CTA layout
	const bool pre = ctx->tune_cg_precond != 0;
	{
		static std::atomic<uint32_t> raised{0};  // one bit per device
		const uint32_t bit = 1u << (ctx->device & 31);
		if (!(raised.load(std::memory_order_acquire) & bit)) {
			for (int pr = 0; pr < 2; pr++)
				for (int sg = 0; sg < 2; sg++)
					for (int per : kCgPerThread) {
						const auto kern = cg_batch_kernel(pr, sg, per);
						NLI_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
						                              (int)kSmemBudget));
						if (!sg)
							NLI_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
					}
			raised.fetch_or(bit, std::memory_order_release);
		}
	}
	for (int ncta = 1; ncta <= kClusterMax; ncta++) {
		CgArgs G;
		std::memset(&G, 0, sizeof(G));
		G.C = C;
		G.ncta = ncta;
		G.active = active;
		G.timeout = &ctx->status->timeout;
		int maxchunk = 0;
		for (int t = 0; t < P.n; t++) {
			const BTask &T = P.t[t];
			if (T.ncta != ncta || T.nh == 0) continue;
			CgTask &g = G.t[G.n++];
			g.img_index = T.img_index;
			g.a = T.pa;
			g.chunk = T.chunk;
			g.unk = T.unkc;
			g.b = T.b;
			g.x0 = T.x;
			g.iters = T.iters;
			g.hole = T.hole;
			g.orig = T.orig;
			g.img = T.img;
			g.diff = T.diff;
			maxchunk = std::max(maxchunk, T.chunk);
		}
		if (G.n == 0) continue;
		const size_t smem = cg_smem_bytes(maxchunk);
		const auto kern = cg_batch_kernel(pre, ncta == 1, cg_per_thread(maxchunk));
		ProfScope ps(ctx, "poisson_cg");
		if (ncta == 1) {
			kern<<<G.n * C, kClusterBlock, smem, s>>>(G);
			NLI_CHECK_LAUNCH();
			continue;
		}
		cudaLaunchConfig_t cfg = {};
		cfg.gridDim = dim3(G.n * C * ncta);
		cfg.blockDim = dim3(kClusterBlock);
		cfg.dynamicSmemBytes = smem;
		cfg.stream = s;
		cudaLaunchAttribute attr[1];
		attr[0].id = cudaLaunchAttributeClusterDimension;
		attr[0].val.clusterDim.x = ncta;
		attr[0].val.clusterDim.y = 1;
		attr[0].val.clusterDim.z = 1;
		cfg.attrs = attr;
		cfg.numAttrs = 1;
		NLI_CUDA(cudaLaunchKernelEx(&cfg, kern, G));
		nli_count_launch_internal();
	}
	// systems too large for a cluster: the cooperative grid CG, one at a time
	for (int t = 0; t < P.n; t++) {
		const BTask &T = P.t[t];
		if (T.ncta != 0 || T.nh == 0) continue;
		const int i = T.img_index;  // names its scratch
		const size_t nh = (size_t)T.nh;
		PoissonSystem S;
		S.pa = T.pa;
		S.co = T.co;
		S.unk = T.unk;
		S.b = T.b;
		S.x = T.x;
		const GridLayout gl = grid_layout(ctx, T.nh, C, T.W);
		if (gl.groups > 0) {
			launch_wide_cg(ctx, S, gl, T.iters, T.hole, T.orig, T.img, T.diff,
			               active ? active + T.img_index : nullptr);
			continue;
		}
		GridCgBufs g;
		g.r = ctx->buf<float>(lk_name(i, "r"), nh * C);
		g.d = ctx->buf<float>(lk_name(i, "d"), nh * C);
		g.q = ctx->buf<float>(lk_name(i, "q"), nh * C);
		g.z = pre ? ctx->buf<float>(lk_name(i, "z"), nh * C) : nullptr;
		g.part = ctx->buf<double>(lk_name(i, "part"), (size_t)T.nparts * 16);
		launch_grid_cg(ctx, S, T.nparts, g, T.iters, T.hole, T.orig, T.img, T.diff,
		               active ? active + T.img_index : nullptr);
	}
	k_total_batch<<<P.n, 1024, 0, s>>>(P, 1);
	NLI_CHECK_LAUNCH();
}

// ============================================================== adjoints
// Backward of one image update with the NNF held fixed: out = U(u; lambda,
// sigma) with orig = u (the update step of image_inpainting.cpp:394 on its
// own), given g = dL/dout.  The NNF is an integer argmin and is not
// differentiated.  Accumulation into dL/du is in double (atomics), then
// rounded to float.  sigma enters through the normalised Gaussian patch
// weights w_k = e_k / sum_j e_j, e_k = exp(-r_k^2 / (2 sigma^2))
// (gaussian_weights.cpp:19-79): dw_k/dsigma = w_k (rho_k - m), rho_k =
// r_k^2 / sigma^3, m = sum_j w_j rho_j.
// The factor rho_k - m per tap as a pair of floats, formed once on the host and
// scaled by a power of two so that the largest is near 1 (at sigma 1e13 they are
// below the smallest float): the kernels' dL/dsigma are scaled so too.
struct AdjArgs {
	float2 rho_m[kMaxTaps];
};

// dL/du is accumulated by channel (element (p, c) at c * W * H + p): the threads
// of a warp then add to neighbouring words where their pixels are neighbours.
// Identity part: out = u outside the domain (and on domain pixels without
// any valid candidate, handled by the means kernel).
__global__ void k_adj_init(const float *__restrict__ g, const uint8_t *__restrict__ dom, int n, int C,
                           double *__restrict__ gacc)
{
	for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n * C; i += gridDim.x * blockDim.x)
		gacc[(size_t)(i % C) * n + i / C] = dom[i / C] ? 0.0 : (double)g[i];
}


// NL-Poisson, per pixel q: the adjoints of the coefficients S(q), U(q),
// GX(q), GY(q) for the residual F_k = lambda U_k - (1-lambda) D_k -
// lambda S_k out_k + (1-lambda) sum_nb s_nb(k) (out_nb - out_k) (D = the
// backward divergence of (GX, GY), s_up / s_left = S of that neighbour,
// s_down / s_right = S_k), weighted by the adjoint solution z = A^-1 g on
// the hole; the boundary-coupling part of dL/du for pixels outside the
// hole; and dL/dlambda per hole pixel.
struct AdjCoef {
	float *dS;   // W*H
	float *dU;   // W*H*C
	float *dGX;  // W*H*C
	float *dGY;  // W*H*C
};

__global__ void k_poisson_adj_coef(PoissonArgs pa, CoefOut co, AdjCoef ad, const uint8_t *__restrict__ dom,
                                   const float *__restrict__ out, const float *__restrict__ z,
                                   double *__restrict__ gacc,
                                   double *__restrict__ lam_part, int depth)
{
	__shared__ double red[2][8];
	const int W = pa.W, H = pa.H, C = pa.C;
	const int q = blockIdx.x * blockDim.x + threadIdx.x;
	double dl = 0.0, dld = 0.0;
	if (q < W * H) {
		const int x = q % W, y = q / W;
		const bool hq = dom[q] != 0;
		const bool hr = (x != W - 1) && dom[q + 1];
		const bool hd = (y != H - 1) && dom[q + W];
		const bool hl = (x != 0) && dom[q - 1];
		const bool hu = (y != 0) && dom[q - W];
		const bool act = hq || hr || hd;
		float dS = 0.f;
		for (int c = 0; c < C; c++) {
			const float lam = pa.lambda[c], oml = 1.0f - lam;
			const size_t o = (size_t)C * q + c;
			const float zq = hq ? z[o] : 0.f;
			const float zr = hr ? z[o + C] : 0.f;
			const float zd = hd ? z[o + (size_t)C * W] : 0.f;
			const float oq = out[o];
			if (act) {
				ad.dU[o] = lam * zq;
				ad.dGX[o] = (x != W - 1) ? oml * (zr - zq) : 0.f;
				ad.dGY[o] = (y != H - 1) ? oml * (zd - zq) : 0.f;
				float s = 0.f;
				if (hq) {
					s -= lam * oq;
					if (y != H - 1) s += oml * (out[o + (size_t)C * W] - oq);
					if (x != W - 1) s += oml * (out[o + C] - oq);
					s *= zq;
				}
				if (hd) s += zd * oml * (oq - out[o + (size_t)C * W]);
				if (hr) s += zr * oml * (oq - out[o + C]);
				dS += s;
			}
			if (hq) {
				// dF_k / dlambda
				const float Sk = co.S[q];
				float Dk = 0.f;
				if (x != W - 1) Dk += co.GX[o];
				if (x != 0) Dk -= co.GX[o - C];
				if (y != H - 1) Dk += co.GY[o];
				if (y != 0) Dk -= co.GY[o - (size_t)C * W];
				float lap = 0.f;
				if (y != 0) lap += co.S[q - W] * (out[o - (size_t)C * W] - oq);
				if (x != 0) lap += co.S[q - 1] * (out[o - C] - oq);
				if (y != H - 1) lap += Sk * (out[o + (size_t)C * W] - oq);
				if (x != W - 1) lap += Sk * (out[o + C] - oq);
				const double v = (double)zq * ((double)co.U[o] + Dk - (double)Sk * oq - lap);
				if (depth && c == 3)
					dld += v;
				else
					dl += v;
			} else {
				// the coupling into the hole's stencil, (1 - lambda) sum over
				// hole neighbours k of z_k s_q(k) (the identity part, g, is
				// already in gacc from k_adj_init)
				double v = 0.0;
				if (hd) v += (double)oml * z[o + (size_t)C * W] * co.S[q];       // q is the upper neighbour of k
				if (hu) v += (double)oml * z[o - (size_t)C * W] * co.S[q - W];   // q is the lower neighbour
				if (hr) v += (double)oml * z[o + C] * co.S[q];                   // q is the left neighbour
				if (hl) v += (double)oml * z[o - C] * co.S[q - 1];               // q is the right neighbour
				if (v != 0.0) atomicAdd(gacc + (size_t)c * W * H + q, v);
			}
		}
		if (act) ad.dS[q] = dS;
	}
	dl = block_sum<256>(dl, red[0]);
	dld = block_sum<256>(dld, red[1]);
	if (threadIdx.x == 0) {
		lam_part[2 * blockIdx.x] = dl;
		lam_part[2 * blockIdx.x + 1] = dld;
	}
}

// A sum of products kept as a pair of floats.
__device__ __forceinline__ void pair_add(float2 &s, float2 v)
{
	const float t = s.x + v.x, b = t - s.x;
	s.y += ((s.x - (t - b)) + (v.x - b)) + v.y;
	s.x = t;
}

__device__ __forceinline__ float2 pair_mul(float2 a, float2 b)
{
	const float p = fm(a.x, b.x);
	return make_float2(p, fmaf(a.x, b.x, -p) + fmaf(a.x, b.y, fm(a.y, b.x)));
}

// NL-means: out_c(p) = N_c / D, N_c = sum_i w_i u_c(s_i), D = sum_i w_i, with
// the forward's weights (clipped-corner table index, confidence inside the
// domain).  du(s_i) += g_c w_i / D; dsigma += sum_c g_c sum_i w_i (rho_i - m)
// (u_c(s_i) - out_c) / D (any constant m: the normalisation term cancels in
// the ratio).  A warp per hole pixel, a tap per lane: as one thread per pixel a
// small hole filled a few SMs with chains of 2 x 81 dependent gathers and six
// FP64 operations per tap and channel.  The sums are pairs of floats (48 bits), one
// product per atomic is left in double.  Forward and backward of 512 x 512 take
// 550 us instead of 954, of 66 x 68 454 instead of 700 (most of what is left is
// launches and waits of the host); the error against 64 bits falls from 1e-6 to
// 2e-7 for dL/du and from 5e-6 relative to 1e-8 for dL/dsigma, as the sum of the
// weights is no longer rounded tap by tap.
template <int C>
__global__ void __launch_bounds__(256) k_means_backward(UpdArgs u, const __grid_constant__ AdjArgs a,
                                                        const float *__restrict__ img,
                                                        const int32_t *__restrict__ hole, int nh,
                                                        const uint8_t *__restrict__ dom, const int2 *__restrict__ nnf,
                                                        const float *__restrict__ conf, const float *__restrict__ g,
                                                        double *__restrict__ gacc, double *__restrict__ partials)
{
	__shared__ double red[8];
	// the lanes' taps differ: tables in shared memory, not in the constant bank
	__shared__ float s_w[kMaxTaps];
	__shared__ float2 s_rho[kMaxTaps];
	const int lane = threadIdx.x & 31, W = u.W, H = u.H;
	for (int t = threadIdx.x; t < min(2 * u.hy * u.px + 2 * u.hx + 1, kMaxTaps); t += blockDim.x) {
		s_w[t] = u.weights[t];
		s_rho[t] = a.rho_m[t];
	}
	__syncthreads();
	double dsig = 0.0;
	for (int i = blockIdx.x * 8 + (threadIdx.x >> 5); i < nh; i += gridDim.x * 8) {
		const int pix = hole[i];
		const int x = pix % W, y = pix / W;
		const int x_a = max(x - u.hx, 0), nx = min(x + u.hx, W - 1) - x_a + 1;
		const int y_a = max(y - u.hy, 0), taps = nx * (min(y + u.hy, H - 1) - y_a + 1);
		// tap t of the window: its source pixel (-1: none), table index, weight
		auto tap = [&](int t, int &k, float &w) {
			const int dy = t / nx, dx = t - dy * nx;
			const int ii = x_a + dx, jj = y_a + dy;
			const int2 q = nnf[jj * W + ii];
			const int sx = q.x + x - ii, sy = q.y + y - jj;
			if (q.x == -1 || sx < 0 || sy < 0 || sx >= W || sy >= H) return -1;
			k = dy * u.px + dx;
			w = s_w[k];
			if (conf && dom[jj * W + ii]) w = fm(w, conf[jj * W + ii]);
			return sy * W + sx;
		};
		float2 tw = make_float2(0.f, 0.f), tv[C];
#pragma unroll
		for (int c = 0; c < C; c++) tv[c] = tw;
		int k = 0;
		float w = 0.f, most = 0.f;  // the largest value
		for (int t = lane; t < taps; t += 32) {
			const int src = tap(t, k, w);
			if (src < 0) continue;
			pair_add(tw, make_float2(w, 0.f));
#pragma unroll
			for (int c = 0; c < C; c++) {
				const float v = img[(size_t)C * src + c], p = fm(v, w);
				pair_add(tv[c], make_float2(p, fmaf(v, w, -p)));
				most = fmaxf(most, fabsf(v));
			}
		}
		most = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(most)));
#pragma unroll
		for (int o = 16; o > 0; o >>= 1) {
			pair_add(tw, make_float2(__shfl_xor_sync(0xffffffffu, tw.x, o), __shfl_xor_sync(0xffffffffu, tw.y, o)));
#pragma unroll
			for (int c = 0; c < C; c++)
				pair_add(tv[c], make_float2(__shfl_xor_sync(0xffffffffu, tv[c].x, o),
				                            __shfl_xor_sync(0xffffffffu, tv[c].y, o)));
		}
		const float *gp = g + (size_t)C * pix;
		if (!(tw.x > 0.0f)) {
			if (lane < C) atomicAdd(gacc + (size_t)lane * W * H + pix, (double)gp[lane]);
			continue;
		}
		if (!(tw.x >= 0x1p-30f && tw.x <= 0x1p60f && (most == 0.f || (most >= 0x1p-60f && most <= 0x1p60f)))) {
			// weights or values so small or large that the pairs lose bits or
			// overflow (a pixel whose only matches lie where the patch weight is
			// subnormal, a confidence near 0): the same in doubles
			double D = 0.0, N[C];
#pragma unroll
			for (int c = 0; c < C; c++) N[c] = 0.0;
			for (int t = lane; t < taps; t += 32) {
				const int src = tap(t, k, w);
				if (src < 0) continue;
				D += (double)w;
#pragma unroll
				for (int c = 0; c < C; c++) N[c] += (double)w * img[(size_t)C * src + c];
			}
			const double inv = 1.0 / __shfl_sync(0xffffffffu, warp_sum(D), 0);
#pragma unroll
			for (int c = 0; c < C; c++) N[c] = __shfl_sync(0xffffffffu, warp_sum(N[c]), 0) * inv;
			for (int t = lane; t < taps; t += 32) {
				const int src = tap(t, k, w);
				if (src < 0) continue;
				const double wd = (double)w * inv, dw = wd * ((double)s_rho[k].x + (double)s_rho[k].y);
#pragma unroll
				for (int c = 0; c < C; c++) {
					atomicAdd(gacc + (size_t)c * W * H + src, (double)gp[c] * wd);
					dsig += (double)gp[c] * dw * ((double)img[(size_t)C * src + c] - N[c]);
				}
			}
			continue;
		}
		// 1 / D to second order, and the output
		const float inv = __frcp_rn(tw.x);
		const float rest = fm(inv, fmaf(-inv, tw.y, fmaf(-inv, tw.x, 1.0f)));
		const double inv_d = (double)inv + (double)rest;
		float2 out[C], acc[C];
		double gd[C];
#pragma unroll
		for (int c = 0; c < C; c++) {
			out[c] = pair_mul(tv[c], make_float2(inv, rest));
			acc[c] = make_float2(0.f, 0.f);
			gd[c] = (double)gp[c] * inv_d;
		}
		for (int t = lane; t < taps; t += 32) {
			const int src = tap(t, k, w);
			if (src < 0) continue;
			const float2 dw = pair_mul(make_float2(w, 0.f), s_rho[k]);
#pragma unroll
			for (int c = 0; c < C; c++) {
				atomicAdd(gacc + (size_t)c * W * H + src, gd[c] * (double)w);
				float2 d = make_float2(img[(size_t)C * src + c], 0.f);
				pair_add(d, make_float2(-out[c].x, -out[c].y));
				pair_add(acc[c], pair_mul(dw, d));
			}
		}
#pragma unroll
		for (int c = 0; c < C; c++) dsig += gd[c] * ((double)acc[c].x + (double)acc[c].y);
	}
	dsig = block_sum<256>(dsig, red);
	if (threadIdx.x == 0) partials[blockIdx.x] = dsig;
}

// Scatter of the coefficient adjoints through the gathers of
// k_poisson_coef: for every coefficient pixel q and every extended-domain
// centre c of its window with n = nnf(c) + q - c in the image,
//   du(n) += w dU(q), gx / gy of n (forward differences of u) take w dGX(q),
//   w dGY(q), and dsigma += dw/dsigma (dS(q) + sum_c dU u(n) + dGX gx(n) +
//   dGY gy(n)).
// Where the field is coherent, consecutive taps of a window name the same n:
// their weights (and weights times rho - m) are first added up, as pairs of
// floats (exact to 2^-43; FP64 is a sixty-fourth of the FP32 rate here, and what
// is left of it still bounds the kernel where the field is rough), and n is read and its up to nine double atomics
// issued once per run of taps.  One thread per coefficient pixel, the hole
// pixels first (as k_poisson_coef8's items).  With a thread per image pixel, every
// tap on its own and rho_k by a double division a 512 x 512 step took 1248 us
// (29 million atomics), with the runs but their sums in double 534 us; this
// takes 294 us.
template <int C>
__global__ void __launch_bounds__(128) k_poisson_adj_scatter(UpdArgs u, const __grid_constant__ AdjArgs a, AdjCoef ad,
                                                             const int32_t *__restrict__ hole, int nh,
                                                             const uint8_t *__restrict__ dom,
                                                             const uint8_t *__restrict__ ext,
                                                             const int2 *__restrict__ nnf,
                                                             const float *__restrict__ conf,
                                                             const float4 *__restrict__ pad,
                                                             double *__restrict__ gacc, double *__restrict__ partials)
{
	__shared__ double red[4];
	const int W = u.W, H = u.H;
	const int item = blockIdx.x * blockDim.x + threadIdx.x;
	double dsig = 0.0;
	int qx = 0, qy = 0;
	bool owned = item < 3 * nh;
	if (owned) {
		const int pix = hole[item < nh ? item : (item - nh) >> 1];
		qx = pix % W, qy = pix / W;
		if (item >= nh) {
			if (((item - nh) & 1) == 0) {
				owned = qx > 0 && !dom[pix - 1];
				qx--;
			} else {
				owned = qy > 0 && !dom[pix - W] && !(qx + 1 < W && dom[pix - W + 1]);
				qy--;
			}
		}
	}
	if (owned) {
		const int q = qy * W + qx;
		float dU[C], dGX[C], dGY[C];
#pragma unroll
		for (int c = 0; c < C; c++) {
			dU[c] = ad.dU[(size_t)C * q + c];
			dGX[c] = ad.dGX[(size_t)C * q + c];
			dGY[c] = ad.dGY[(size_t)C * q + c];
		}
		const float dS = ad.dS[q];
		int run = -1;                   // the run's source pixel
		float2 wsum = make_float2(0.f, 0.f), dsum = wsum;  // of w and of dw/dsigma
		float2 sig = wsum;                                 // the pixel's share of dL/dsigma
		auto flush = [&]() {
			const int nx = run % W, ny = run / W;
			const Pix3 t3 = load_pix3(pad, W, H, nx, ny);
			const float v[4] = {t3.v.x, t3.v.y, t3.v.z, t3.v.w}, gx[4] = {t3.gx.x, t3.gx.y, t3.gx.z, t3.gx.w};
			const float gy[4] = {t3.gy.x, t3.gy.y, t3.gy.z, t3.gy.w};
			const double w = (double)wsum.x + (double)wsum.y;
			Dot2 t;
			t.h = dS;
#pragma unroll
			for (int c = 0; c < C; c++) {
				double *at = gacc + (size_t)c * W * H + run;
				t.add(dU[c], v[c]);
				t.add(dGX[c], gx[c]);
				t.add(dGY[c], gy[c]);
				double own = w * dU[c];
				if (nx != W - 1) {
					const double g = w * dGX[c];
					atomicAdd(at + 1, g);
					own -= g;
				}
				if (ny != H - 1) {
					const double g = w * dGY[c];
					atomicAdd(at + W, g);
					own -= g;
				}
				atomicAdd(at, own);
			}
			pair_add(sig, pair_mul(dsum, make_float2(t.h, t.l)));
			wsum = dsum = make_float2(0.f, 0.f);
		};
		const int cy0 = max(qy - u.hy, 0), cy1 = min(qy + u.hy, H - 1);
		const int cx0 = max(qx - u.hx, 0), cx1 = min(qx + u.hx, W - 1);
		for (int cy = cy0; cy <= cy1; cy++)
			for (int cx = cx0; cx <= cx1; cx++) {
				const int c0 = cy * W + cx;
				if (!ext[c0]) continue;
				const int2 nb = nnf[c0];
				const int nx = nb.x + qx - cx, ny = nb.y + qy - cy;
				if (nx < 0 || ny < 0 || nx >= W || ny >= H) continue;
				const int k = (qy - cy + u.hy) * u.px + (qx - cx + u.hx);
				const int n = ny * W + nx;
				if (n != run) {
					if (run >= 0) flush();
					run = n;
				}
				const float cf = conf ? conf[c0] : 1.0f, wk = u.weights[k];
				const float p = fm(cf, wk);
				const float2 w = make_float2(p, fmaf(cf, wk, -p));
				pair_add(wsum, w);
				pair_add(dsum, pair_mul(w, a.rho_m[k]));
			}
		if (run >= 0) flush();
		dsig = (double)sig.x + (double)sig.y;
	}
	dsig = block_sum<128>(dsig, red);
	if (threadIdx.x == 0) partials[blockIdx.x] = dsig;
}

__global__ void k_hole_to_planar(const float *__restrict__ g, const int32_t *__restrict__ hole, int nh, int C,
                                 float *__restrict__ b)
{
	const int i = blockIdx.x * blockDim.x + threadIdx.x;
	if (i >= nh * C) return;
	const int k = i % nh, c = i / nh;
	b[i] = g[(size_t)C * hole[k] + c];
}

__global__ void k_to_float(const double *__restrict__ a, int n, int C, float *__restrict__ out)
{
	for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n * C; i += gridDim.x * blockDim.x)
		out[i] = (float)a[(size_t)(i % C) * n + i / C];
}

static double sum_on_host(nli_ctx *ctx, const double *partials, int n, int stride, int offset)
{
	std::vector<double> h((size_t)n * stride);
	NLI_CUDA(cudaMemcpyAsync(h.data(), partials, sizeof(double) * h.size(), cudaMemcpyDeviceToHost, ctx->stream));
	NLI_CUDA(cudaStreamSynchronize(ctx->stream));
	double s = 0.0;
	for (int i = 0; i < n; i++) s += h[(size_t)i * stride + offset];
	return s;
}

void update_backward_run(nli_ctx *ctx, const nli_update_params &up, const float *image, const float *out,
                         const uint8_t *dom, const uint8_t *ext, const int32_t *nnf_i, const float *conf, int W,
                         int H, int C, const float *grad_out, float *grad_image, double *grad_lambda,
                         double *grad_lambda_d, double *grad_sigma)
{
	NLI_REQUIRE(up.method == NLI_UPDATE_MEANS || up.method == NLI_UPDATE_POISSON || up.method == NLI_UPDATE_DEPTH,
	            NLI_E_UNSUPPORTED, "no adjoint for this update method (the weighted median is piecewise constant)");
	if (up.method == NLI_UPDATE_DEPTH) NLI_REQUIRE(C == 4, NLI_E_CHANNELS, "Separate: Channels do not match.");
	UpdArgs u;
	fill_upd_args(u, up, W, H, C);
	AdjArgs a;
	std::memset(&a, 0, sizeof(a));
	const double sigma3 = (double)up.sigma * up.sigma * up.sigma;
	double rho[kMaxTaps], m = 0.0;
	for (int k = 0; k < kMaxTaps; k++) {
		const int kx = k % u.px - u.hx, ky = k / u.px - u.hy;
		// a tap without weight counts for nothing, whatever its factor
		rho[k] = u.weights[k] != 0.f ? (double)(kx * kx + ky * ky) / sigma3 : 0.0;
		if (k < u.px * u.py) m += (double)u.weights[k] * rho[k];
	}
	double most = 0.0;
	for (int k = 0; k < kMaxTaps; k++) most = std::max(most, std::fabs(rho[k] - m));
	const int exponent = most > 0.0 && std::isfinite(most) ? std::ilogb(most) : 0;
	for (int k = 0; k < kMaxTaps; k++) {
		const double d = std::ldexp(rho[k] - m, -exponent);
		a.rho_m[k].x = (float)d;
		a.rho_m[k].y = (float)(d - (double)a.rho_m[k].x);
	}
	cudaStream_t s = ctx->stream;
	const size_t n = (size_t)W * H;
	const int2 *nnf = reinterpret_cast<const int2 *>(nnf_i);
	int32_t *hole = ctx->buf<int32_t>("adj.hole", n);
	const int nh = compact_mask(ctx, dom, W, H, hole, "adj");
	double *gacc = ctx->buf<double>("adj.gacc", n * C);
	k_adj_init<<<(int)std::min<size_t>((n * C + 255) / 256, 8192), 256, 0, s>>>(grad_out, dom, (int)n, C, gacc);
	NLI_CHECK_LAUNCH();
	*grad_lambda = 0.0;
	*grad_lambda_d = 0.0;
	*grad_sigma = 0.0;
	if (nh > 0 && up.method == NLI_UPDATE_MEANS) {
		const int grid = std::min((nh + 7) / 8, 8 * ctx->num_sms);
		double *part = ctx->buf<double>("adj.part", grid);
		with_channels(C, [&](auto c) {
			k_means_backward<decltype(c)::value><<<grid, 256, 0, s>>>(u, a, image, hole, nh, dom, nnf, conf, grad_out,
			                                                          gacc, part);
			NLI_CHECK_LAUNCH();
		});
		*grad_sigma = std::ldexp(sum_on_host(ctx, part, grid, 1, 0), exponent);
	} else if (nh > 0) {
		// system of the forward step with orig = image; its right-hand side
		// is replaced by g on the hole, and z = A^-1 g is written as an image
		PoissonSystem P = poisson_system(ctx, u, up, image, image, dom, ext, nnf, conf, hole, nh);
		k_hole_to_planar<<<(nh * C + 255) / 256, 256, 0, s>>>(grad_out, hole, nh, C, P.b);
		NLI_CHECK_LAUNCH();
		NLI_CUDA(cudaMemsetAsync(P.x, 0, sizeof(float) * nh * C, s));
		float *zimg = ctx->buf<float>("adj.z", n * C);
		float *zero = ctx->buf<float>("adj.zero", n * C);
		NLI_CUDA(cudaMemsetAsync(zimg, 0, sizeof(float) * n * C, s));
		NLI_CUDA(cudaMemsetAsync(zero, 0, sizeof(float) * n * C, s));
		const int np = poisson_solve(ctx, P, hole, zero, zimg);
		(void)read_total(ctx, ctx->buf<double>("poi.diff", np + 1), np, ctx->buf<int>("poi.iters", 4), C, nh);
		AdjCoef ad;
		ad.dS = ctx->buf<float>("adj.dS", n);
		ad.dU = ctx->buf<float>("adj.dU", n * C);
		ad.dGX = ctx->buf<float>("adj.dGX", n * C);
		ad.dGY = ctx->buf<float>("adj.dGY", n * C);
		const int grid = (int)((n + 255) / 256);
		double *lam_part = ctx->buf<double>("adj.lam", 2 * (size_t)grid);
		k_poisson_adj_coef<<<grid, 256, 0, s>>>(P.pa, P.co, ad, dom, out, zimg, gacc, lam_part,
		                                        up.method == NLI_UPDATE_DEPTH ? 1 : 0);
		NLI_CHECK_LAUNCH();
		const int grid2 = (3 * nh + 127) / 128;
		double *sig_part = ctx->buf<double>("adj.sig", grid2);
		with_channels(C, [&](auto c) {
			k_poisson_adj_scatter<decltype(c)::value><<<grid2, 128, 0, s>>>(u, a, ad, hole, nh, dom, ext, nnf, conf, P.pad,
			                                                                 gacc, sig_part);
			NLI_CHECK_LAUNCH();
		});
		*grad_lambda = sum_on_host(ctx, lam_part, grid, 2, 0);
		*grad_lambda_d = sum_on_host(ctx, lam_part, grid, 2, 1);
		*grad_sigma = std::ldexp(sum_on_host(ctx, sig_part, grid2, 1, 0), exponent);
	}
	k_to_float<<<(int)std::min<size_t>((n * C + 255) / 256, 8192), 256, 0, s>>>(gacc, (int)n, C, grad_image);
	NLI_CHECK_LAUNCH();
	NLI_CUDA(cudaStreamSynchronize(s));
}

}  // namespace nli
