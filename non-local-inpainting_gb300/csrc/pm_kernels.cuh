// PatchMatch::calculate (patch_match.cpp:311-512) as data-parallel sweeps.
//
// The reference visits target points in scanline order and lets each point
// see the matches its predecessors found in the same sweep.  Here every
// target point of a sweep is updated at once from the field of the previous
// sweep (a Jacobi sweep, so results do not depend on thread timing):
//   1. propagation: the matches of the 4 neighbours at distance 1 and of the
//      4 neighbours at a jump distance J (J = 16, 8, 4, 2, ... by sweep),
//      each shifted back by the neighbour's offset (the reference tries the
//      left/upper or right/lower neighbour at distance 1, :420-451);
//   2. random search around the best match after propagation, in windows
//      max(W,H), /2, ..., 1 with up to `random_shots` draws per window and
//      the first draw that lands in the source evaluated (:458-494).
// A candidate equal to the current match, or to an earlier candidate of the
// same step, is not re-evaluated (its distance would not be smaller).
// Random draws come from Philox4x32-10 keyed by the context seed and call
// counter.
//
// Layout and work split.  Images are read as one float4 per pixel (the C
// channels, zero-filled), with one extra column and row that repeat the
// last ones, so the forward differences u(x+1) - u(x) and u(y+1) - u(y) are
// exactly 0 on the last column / row, as Gradient::calculate sets them
// (gradient.cpp:37-63).
//
// A warp works on a group of up to three target points at a time.  To
// propose, its lanes are split evenly over the points (10, 16 or 32 lanes
// each): a point's lanes each fetch one neighbour's match, or draw in one
// random-search window, test it and drop it where the lower bound below
// rules it out.  What survives goes into one list for the whole warp, in
// the order of points and proposals.  To evaluate, the lanes are split into
// K = 32 / L sub-warps of L = patch width + 1 lanes (3 sub-warps of 10 lanes
// for 9x9 patches), and each round takes the next K entries of the list,
// whichever points they belong to.  In a sub-warp lane c walks down column c
// of the candidate's and the target's window: per row it loads one float4
// of each, forms the colour difference d = u_s - u_t, gets d of column c + 1
// by a shuffle (x gradient difference) and keeps the previous row's d in
// registers (y gradient difference).  The gradient difference of the two
// patches is formed as a difference of colour differences,
// (u_s(x+1) - u_t(x+1)) - (u_s(x) - u_t(x)), which equals (gx_s - gx_t) up to
// float rounding.  Results are accepted in the list's order with a strict
// "<", so the field equals evaluating each point's candidates one after the
// other, whatever the grouping.  Where a call has too few points to fill
// the SMs it is the other way round: two or four warps share a point
// (k_pm_sweep_team).
//
// Why groups: in a run whose field has converged about two of a point's
// eighteen proposals survive the bound, so one point filled two of the three
// sub-warps in a round of its own, and its proposing (the random draws, the
// mask tests and the bound, over 500 instructions) kept 8 to 10 of 32 lanes
// busy.  Three points share both: a call on
// 512 x 512 takes 1466 us instead of 1567, on 1013 x 887 5720 instead of 6847,
// on 640 x 480 RGB-D 1695 instead of 2035 (figures of the bound by means).
#pragma once

#include <cuda.h>  // CUtensorMap (the descriptor type; encoded through the runtime's driver entry point)

#include <atomic>
#include <type_traits>

#include "nli_device.cuh"

namespace nli {

constexpr unsigned kFull = 0xffffffffu;

// ------------------------------------------------------- TMA staging
// With 9 x 9 patches each candidate's source window (rows x L float4) is
// copied into the warp's shared memory by one tensor copy
// (cp.async.bulk.tensor.2d) instead of being read row by row through L1.
// The copies of a step complete on the warp's mbarrier; waiting is bounded
// and a wait that runs out sets the context's timeout flag.
constexpr unsigned kTmaWaitLimit = 1u << 22;

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t *bar, unsigned count)
{
	asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
	asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, unsigned bytes)
{
	asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, unsigned parity)
{
	uint32_t ok;
	asm volatile(
	    "{\n\t.reg .pred p;\n\t"
	    "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
	    "selp.u32 %0, 1, 0, p;\n\t}"
	    : "=r"(ok)
	    : "r"(smem_u32(bar)), "r"(parity)
	    : "memory");
	return ok != 0;
}

// Bounded wait for the phase `parity` of the barrier; false when it ran out.
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, unsigned parity)
{
	for (unsigned i = 0; i < kTmaWaitLimit; i++)
		if (mbar_try_wait(bar, parity)) return true;
	return false;
}

// Orders this thread's earlier generic-proxy accesses of shared memory
// before later async-proxy (tensor copy) writes to it.
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// Tile [x, x + box0) x [y, y + box1) of the 2-D tensor into dst; x counts
// floats and is a multiple of 4 (16 bytes) here.
__device__ __forceinline__ void tma_load_2d(void *dst, const CUtensorMap *map, int x, int y, uint64_t *bar)
{
	asm volatile(
	    "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
	        smem_u32(dst)),
	    "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(smem_u32(bar))
	    : "memory");
}

// How the fixed-size (9 x 9) kernels work (NLI_TUNE_PM_VARIANT): kPmGrouped
// (the default, described above) takes groups of points and loads both
// windows' rows from global memory.  The other two take one point per warp:
// kPmStaged keeps the target window in shared memory and copies the source
// windows there by tensor copies; kPmRegs holds the lane's column of the
// target window in registers (16 warps per SM, twice the registers).  All
// three evaluate the same candidates with the same arithmetic.
// Runtime-sized patches and batches always use kPmGrouped.
enum PmVariant { kPmGrouped = 0, kPmStaged = 1, kPmRegs = 2 };

__host__ __device__ constexpr int pm_threads(int V) { return V == kPmRegs ? 512 : 1024; }

// Lanes per target point and points per warp when a warp proposes: enough
// lanes for a call's random-search windows (max_window, max_window / 2, ...,
// 1: 10 up to sides of 1023) and for its 8 neighbours.
struct PmGroup {
	int lanes, points;
};

// Launch shape of the persistent kernels for `items` work items (groups of
// points, or points): one block per SM, with just enough warps that every
// item has one (up to the variant's most).  An item is one warp's serial
// chain of loads and evaluations, and a sweep of a coarse level is bound by
// the warps that share an SM, so the items are spread over all SMs first: a
// PatchMatch call on a 64 x 48 level (500 points) took 348 us with full
// blocks on 16 SMs and 288 us with 4 warps on each of 125.
struct PmShape {
	int grid, block;
};

inline PmShape pm_shape(int threads, long long items, int num_sms)
{
	const int most = threads / 32;
	const long long per_sm = (items + num_sms - 1) / num_sms;
	const int warps = (int)std::max(1LL, std::min((long long)most, per_sm));
	return {(int)std::min((long long)num_sms, (items + warps - 1) / warps), 32 * warps};
}

// Groups for a call of nt points in all.  Several points per group take
// fewer instructions per point but make a warp's chain of rounds longer, so
// they pay once every SM has 16 groups: 512 x 512 (50 000 points) 1715 us a
// call with one point per group and 1466 us with three, 276 x 167 RGB-D
// (11 000) 569 and 510 us, but 64 x 48 (750) 296 and 416 us, 190 x 107 (6500)
// 457 and 542 us.  The line lies near 7300 points: 8 or 24 groups per SM are
// slower on calls of 4000 to 11 000 points.
inline PmGroup pm_group(long long nt, int max_window, int num_sms)
{
	int windows = 0;
	for (unsigned w = (unsigned)max_window; w; w >>= 1) windows++;
	PmGroup g = windows <= 10 ? PmGroup{10, 3} : windows <= 16 ? PmGroup{16, 2} : PmGroup{32, 1};
	while (g.points > 1 && nt < 16LL * num_sms * g.points) g.points--;
	return g;
}

// Per-warp state of the staged path.
struct TmaState {
	const CUtensorMap *map;
	float4 *slots;    // K windows of rows x L float4, each slot_stride float4 apart
	int slot_stride;  // float4
	uint64_t *bar;
	unsigned phase;
	int *timeout;  // context status flag
};

struct PmArgs {
	const float4 *src;  // source pixels, (sW + 1) x (sH + 1), row stride sWp
	const float4 *tgt;  // target pixels, row stride tWp
	const uint8_t *smask;
	const uint8_t *tmask;
	const int32_t *tlist;
	int sW, sH, tW, tH, nt;
	int sWp, tWp;
	int shots, max_window;
	uint64_t seed;                     // the context's seed
	const unsigned long long *calls;   // PatchMatch calls so far, this one included
	// patch extent around a centre: [x - rx, x + ex) x [y - ry, y + ey)
	int rx, ry, ex, ey;
	// lanes per candidate, candidates per warp step, window rows
	int L, K, rows;
	float lambda, lambda_d;
	// patch-statistics lower bound (null: off): the tables of the padded
	// source and target (n = (W + 1)(H + 1) positions: n float4 of weighted
	// patch means, then n pairs of weighted slopes in x and y), and the
	// largest absolute pixel value of the images (as float bits)
	const float4 *smom, *tmom;
	const unsigned *vmax;
	// 1: the bound uses the slopes; 1: behind them follow the weighted
	// standard deviations (of the image and of its forward differences),
	// and the bound uses them too
	int slopes, dev;
	// device work queue (null: static ranges): the call's counters, one
	// per launch (init, then each sweep), zeroed before the init launch;
	// a warp takes `tile` consecutive target points per grab
	unsigned *queue;
	int tile;
	PmGroup group;  // kPmGrouped
};

// Philox key of this PatchMatch call: the seed mixed with the call's index
// (0 for the first call after the seed is set).
__device__ __forceinline__ uint2 pm_key(const PmArgs &p)
{
	const uint64_t call = *p.calls - 1ull;
	const uint64_t k = p.seed ^ (call * 0x9E3779B97F4A7C15ULL);
	return make_uint2((uint32_t)k, (uint32_t)(k >> 32) ^ (uint32_t)call);
}

template <int KIND>
struct Kind {
	static constexpr bool grad = KIND == NLI_DIST_L2_COMBINED || KIND == NLI_DIST_L2_RGBD;
};

// The work items [0, n) of a persistent PatchMatch launch (groups of target
// points, single points in the variants that take them one by one), visited by the
// calling warp (f(i) for each of its items, in increasing order).  Without
// a queue, block b takes the contiguous range [b * chunk, (b + 1) * chunk)
// and its warps interleave over it, so the warps of an SM work on
// neighbouring points and share source neighbourhoods in L1.  With a queue
// (`queue` a counter zeroed before the launch), each warp starts on the `tile`
// items of its own number and then takes `tile` consecutive items per atomic
// grab until the list is exhausted, so warps that drew cheap points take
// more and no SM idles while others finish.
// Every item's computation is independent of which warp does it and when
// (the sweeps read the previous field and the random streams are keyed by
// point), so both give the same field.
template <class F>
__device__ __forceinline__ void pm_for_each(int n, unsigned *queue, int tile, F &&f)
{
	if (queue) {
		const int lane = threadIdx.x & 31;
		const unsigned warps = gridDim.x * (blockDim.x >> 5), taken = warps * (unsigned)tile;
		unsigned base = (blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * (unsigned)tile;
		while (base < (unsigned)n) {
			const int stop = min(n, (int)base + tile);
			for (int i = (int)base; i < stop; i++) f(i);
			if (taken >= (unsigned)n) break;  // every item had a warp
			if (lane == 0) base = taken + atomicAdd(queue, (unsigned)tile);
			base = __shfl_sync(kFull, base, 0);
		}
	} else {
		const int chunk = (n + gridDim.x - 1) / gridDim.x;
		const int end = min(n, (int)(blockIdx.x + 1) * chunk);
		for (int i = blockIdx.x * chunk + (threadIdx.x >> 5); i < end; i += blockDim.x >> 5) f(i);
	}
}

// A source centre is usable when it is in the source mask and its whole
// patch lies in the image (the masks of the inpainting driver guarantee the
// latter through their margin; user masks may not).
__device__ __forceinline__ bool src_inside(const PmArgs &p, int x, int y)
{
	return x >= p.rx && y >= p.ry && x + p.ex <= p.sW && y + p.ey <= p.sH;
}

__device__ __forceinline__ bool src_masked(const PmArgs &p, int x, int y)
{
	return nli_in_bounds((long long)y * p.sW + x, (long long)p.sW * p.sH, kSitePmMask) && p.smask[y * p.sW + x];
}

__device__ __forceinline__ bool src_ok(const PmArgs &p, int x, int y) { return src_inside(p, x, y) && src_masked(p, x, y); }

__device__ __forceinline__ bool tgt_patch_inside(const PmArgs &p, int x, int y)
{
	return x >= p.rx && y >= p.ry && x + p.ex <= p.tW && y + p.ey <= p.tH;
}

// Shared memory: per-tap weights (divided by the patch area) for all warps,
// padded to a float4 boundary, then one 32-entry candidate list and its
// counts per warp (the staged variant's layout: pm_smem_bytes_tma).
__host__ __device__ inline int pm_weight_slots(int taps) { return (taps + 3) / 4; }

__host__ __device__ inline size_t pm_smem_bytes(int taps, int warps)
{
	return sizeof(float4) * (size_t)pm_weight_slots(taps) + sizeof(int) * 36 * warps;
}

__device__ __forceinline__ void load_weights(const DistArgs &a, float *s_w)
{
	const int taps = a.px * a.py;
	const float invP = 1.0f / (float)taps;
	for (int t = threadIdx.x; t < taps; t += blockDim.x) s_w[t] = a.weights[t] * invP;
	__syncthreads();
}

// kPmStaged: the warp's target window, rows x L pixels starting at the patch
// corner.  With up to 3 channels the unused fourth component carries the
// tap's weight (0 outside the patch), so the distance reads one float4 per
// row.
template <int KIND, int C, int P>
__device__ __forceinline__ void load_window(const PmArgs &p, const float *s_w, int x, int y, float4 *s_t)
{
	const int lane = threadIdx.x & 31;
	constexpr int L = P + (Kind<KIND>::grad ? 1 : 0);
	const float4 *T = p.tgt + (size_t)(y - p.ry) * p.tWp + (x - p.rx);
	for (int e = lane; e < L * L; e += 32) {
		const int r = e / L, c = e - r * L;
		float4 v = __ldg(T + (size_t)r * p.tWp + c);
		if (C <= 3) v.w = (r < P && c < P) ? s_w[r * P + c] : 0.f;
		s_t[e] = v;
	}
	__syncwarp();
}

// kPmRegs: the lane's column c of the same window, tw[r] = element r * L + c
// of load_window's, for a fixed P x P patch.
template <int KIND, int C, int P>
__device__ __forceinline__ void load_window_regs(const PmArgs &p, const float *s_w, int x, int y, float4 *tw)
{
	constexpr int L = P + (Kind<KIND>::grad ? 1 : 0);
	const int lane = threadIdx.x & 31;
	const int c = lane - (lane / L) * L;
	const float4 *T = p.tgt + (size_t)(y - p.ry) * p.tWp + (x - p.rx) + c;
#pragma unroll
	for (int r = 0; r < L; r++) {
		float4 v = __ldg(T + (size_t)r * p.tWp);
		if (C <= 3) v.w = (r < P && c < P) ? s_w[r * P + c] : 0.f;
		tw[r] = v;
	}
}

template <int C>
__device__ __forceinline__ float sq3(float4 d)
{
	float n = d.x * d.x;
	if (C > 1) n = fmaf(d.y, d.y, n);
	if (C > 2) n = fmaf(d.z, d.z, n);
	return n;
}

// sum of squares / absolute values over the first C components
template <int C>
__device__ __forceinline__ float sqc(float4 d)
{
	float n = sq3<C>(d);
	if (C > 3) n = fmaf(d.w, d.w, n);
	return n;
}

template <int C>
__device__ __forceinline__ float absc(float4 d)
{
	float n = fabsf(d.x);
	if (C > 1) n += fabsf(d.y);
	if (C > 2) n += fabsf(d.z);
	if (C > 3) n += fabsf(d.w);
	return n;
}

// a - b over the first C components (the others are left 0)
template <int C>
__device__ __forceinline__ float4 subc(float4 a, float4 b)
{
	return make_float4(a.x - b.x, (C > 1) ? a.y - b.y : 0.f, (C > 2) ? a.z - b.z : 0.f, (C > 3) ? a.w - b.w : 0.f);
}

template <int C>
__device__ __forceinline__ float4 shfl_down4(float4 v, int o)
{
	float4 r;
	r.x = __shfl_down_sync(kFull, v.x, o);
	r.y = (C > 1) ? __shfl_down_sync(kFull, v.y, o) : 0.f;
	r.z = (C > 2) ? __shfl_down_sync(kFull, v.z, o) : 0.f;
	r.w = (C > 3) ? __shfl_down_sync(kFull, v.w, o) : 0.f;
	return r;
}

// Sum over the L lanes of each sub-warp, left in its lane c == 0.
__device__ __forceinline__ float subwarp_sum(float v, int c, int L)
{
#pragma unroll
	for (int o = 1; o < 16; o <<= 1) {
		const float u = __shfl_down_sync(kFull, v, o);
		if (c + o < L) v += u;
	}
	return v;
}

// Per-lane sums of one candidate by term: colour and gradient differences
// of the colour channels (n, g) and of the depth channel (nd, gd, L2 RGBD).
struct Acc {
	float n, g, nd, gd;
};

// Contribution of one window row.  d: colour difference of this lane's
// pixel in row r, dp: of the row above; w, wp: their tap weights.
template <int KIND, int C>
__device__ __forceinline__ void row_terms(const float4 d, const float4 dp, float w, float wp, bool tap, bool tap_above,
                                          Acc &A)
{
	if (KIND == NLI_DIST_L1_NORM) {
		if (tap) A.n = fmaf(w, absc<C>(d), A.n);
		return;
	}
	if (KIND == NLI_DIST_L2_NORM) {
		if (tap) A.n = fmaf(w, sqc<C>(d), A.n);
		return;
	}
	// x gradient difference from the lane to the right (column c + 1)
	const float4 dr = shfl_down4<C>(d, 1);
	if (KIND == NLI_DIST_L2_RGBD) {
		if (tap) {
			const float4 gx = subc<4>(dr, d);
			A.n = fmaf(w, sq3<3>(d), A.n);
			A.g = fmaf(w, sq3<3>(gx), A.g);
			A.nd = fmaf(w, d.w * d.w, A.nd);
			A.gd = fmaf(w, gx.w * gx.w, A.gd);
		}
		if (tap_above) {
			const float4 gy = subc<4>(d, dp);
			A.g = fmaf(wp, sq3<3>(gy), A.g);
			A.gd = fmaf(wp, gy.w * gy.w, A.gd);
		}
	} else {
		if (tap) {
			const float4 gx = subc<C>(dr, d);
			A.n = fmaf(w, sqc<C>(d), A.n);
			A.g = fmaf(w, sqc<C>(gx), A.g);
		}
		if (tap_above) {
			const float4 gy = subc<C>(d, dp);
			A.g = fmaf(wp, sqc<C>(gy), A.g);
		}
	}
}

// The lane's share of the distance: the terms weighted by lambda, 1 - lambda
// (and lambda_d, 1 - lambda_d for the depth channel).
template <int KIND>
__device__ __forceinline__ float combine(const Acc &A, const PmArgs &p)
{
	if (KIND == NLI_DIST_L1_NORM || KIND == NLI_DIST_L2_NORM) return A.n;
	float v = fmaf(p.lambda, A.n, (1.0f - p.lambda) * A.g);
	if (KIND == NLI_DIST_L2_RGBD) v = fmaf(p.lambda_d, A.nd, fmaf(1.0f - p.lambda_d, A.gd, v));
	return v;
}

// float4 helpers of the patch statistics
__device__ __forceinline__ float4 f4_fma(float w, float4 v, float4 a)
{
	return make_float4(fmaf(w, v.x, a.x), fmaf(w, v.y, a.y), fmaf(w, v.z, a.z), fmaf(w, v.w, a.w));
}
__device__ __forceinline__ float4 f4_sub(float4 a, float4 b)
{
	return make_float4(a.x - b.x, a.y - b.y, a.z - b.z, a.w - b.w);
}
__device__ __forceinline__ float4 f4_wsq(float w, float4 d, float4 a)
{
	return make_float4(fmaf(w, d.x * d.x, a.x), fmaf(w, d.y * d.y, a.y), fmaf(w, d.z * d.z, a.z),
	                   fmaf(w, d.w * d.w, a.w));
}
__device__ __forceinline__ float4 f4_sqrt(float4 a)
{
	return make_float4(sqrtf(a.x), sqrtf(a.y), sqrtf(a.z), sqrtf(a.w));
}

// ------------------------------------------------ lower bound
// Jensen's inequality gives, for weights v_k >= 0 summing to V,
//   sum_k v_k |d_k|^2 >= |sum_k v_k d_k|^2 / V,   sum_k v_k |d_k|_1 >= |sum_k v_k d_k|_1.
// With the kernel's tap weights v_k = w_k / P (sum 1 / P) and d_k the colour
// or gradient difference of tap k, sum_k w_k d_k is the difference of the
// two patches' weighted means of the image or of its forward differences;
// the mean of the differences is the difference of means one column (row)
// apart.  So a candidate whose patch means differ enough from the target's
// cannot beat the current match and is not evaluated.
//
// The means are the first of an orthonormal set: with f_0 = 1 and f_1, f_2 the
// centred tap positions in x and y, scaled so that sum_k w_k f_i f_j = (i == j)
// (they are orthogonal because the weights are a product of one factor in x
// and one in y), Bessel's inequality gives
//   sum_k w_k d_k^2 >= sum_j (sum_k w_k f_j d_k)^2.
// The sums of f_1 and f_2, the patch's slopes, are two more linear tables, and
// those of the forward differences are again differences of entries one
// column (row) apart.  The L2 kinds test them (PmArgs::slopes) on what the
// means let through: 686 -> 438 million evaluations in a 512 x 512 NL-Poisson
// process() (590 -> 582 ms), and a first call on 512 x 512 takes 1383 us instead
// of 1466, on 1013 x 887 5385 instead of 5732.
//
// With the weighted standard deviations as well (PmArgs::dev, the L2
// kinds): for weights summing to 1,
//   sum_k w_k d_k^2 = (sum_k w_k d_k)^2 + sum_k w_k (d_k - mean d)^2,
// and with d = s - t the centred part is the squared weighted L2 distance of
// the centred patches, at least (sigma_s - sigma_t)^2 by the reverse
// triangle inequality.  So each channel's colour term is bounded by the
// squared mean difference plus the squared difference of standard
// deviations, and each gradient term likewise with the deviations of the
// forward differences: a second bound beside that of the slopes.
//
// Exactness: every difference of means, slopes and deviations is shrunk by a
// slack (2e-4 of the largest pixel value) that covers the float rounding of
// the tables (sums of 81 products whose weights w_k |f_j| add up to at most
// 1: a few 1e-6 of the largest value) and of the kernel's per-tap
// differences, and the bound must exceed the current distance by a 1e-4
// relative margin that covers the rounding of the kernel's sums and of the
// set's orthonormality; the field and distances are those of evaluating
// every candidate.
__device__ __forceinline__ float shrink(float v, float slack) { return fmaxf(fabsf(v) - slack, 0.f); }

// True when candidate (cx, cy) for target (x, y) provably cannot reach a
// distance below bd.  The target's means are read here too (the same
// address in every lane), so nothing stays live across the evaluations.
template <int KIND, int C>
__device__ __forceinline__ bool bound_rejects(const PmArgs &p, int x, int y, int cx, int cy, float bd)
{
	const float4 *M = p.smom + (size_t)cy * p.sWp + cx;
	const float4 *T = p.tmom + (size_t)y * p.tWp + x;
	const float slack = 2e-4f * __uint_as_float(__ldg(p.vmax));
	// per-channel terms, the depth channel of L2 RGBD kept apart; each
	// statistic is read, folded in and dropped in turn (few live registers)
	float col = 0.f, grad = 0.f, dcol = 0.f, dgrad = 0.f;
	auto add = [&](float4 d, bool g) {
		const float v[4] = {d.x, d.y, d.z, d.w};
#pragma unroll
		for (int c = 0; c < C; c++) {
			const float e = shrink(v[c], slack);
			const bool depth = KIND == NLI_DIST_L2_RGBD && c == 3;
			if (KIND == NLI_DIST_L1_NORM)
				col += e;
			else if (depth)
				(g ? dgrad : dcol) += e * e;
			else
				(g ? grad : col) += e * e;
		}
	};
	const float P = (float)((p.rx + p.ex) * (p.ry + p.ey));
	auto exceeds = [&]() {
		float lb = col;
		if (Kind<KIND>::grad) lb = fmaf(p.lambda, col, (1.0f - p.lambda) * grad);
		if (KIND == NLI_DIST_L2_RGBD) lb = fmaf(p.lambda_d, dcol, fmaf(1.0f - p.lambda_d, dgrad, lb));
		return lb * (1.0f - 1e-4f) >= bd * P;
	};
	const float4 m0 = f4_sub(__ldg(M), __ldg(T));
	add(m0, false);
	if (Kind<KIND>::grad) {
		// the mean of the forward differences: means one column (row) apart
		add(f4_sub(f4_sub(__ldg(M + 1), __ldg(T + 1)), m0), true);
		add(f4_sub(f4_sub(__ldg(M + p.sWp), __ldg(T + p.tWp)), m0), true);
	}
	if (exceeds()) return true;
	if (KIND == NLI_DIST_L1_NORM) return false;
	const size_t sn = (size_t)p.sWp * (p.sH + 1), tn = (size_t)p.tWp * (p.tH + 1);
	if (p.dev) {
		// weighted standard deviations: of the image, of its x and y differences
		const float c0 = col, g0 = grad, d0 = dcol, e0 = dgrad;
		add(f4_sub(__ldg(M + 3 * sn), __ldg(T + 3 * tn)), false);
		if (Kind<KIND>::grad) {
			add(f4_sub(__ldg(M + 4 * sn), __ldg(T + 4 * tn)), true);
			add(f4_sub(__ldg(M + 5 * sn), __ldg(T + 5 * tn)), true);
		}
		if (exceeds()) return true;
		col = c0, grad = g0, dcol = d0, dgrad = e0;
	}
	if (!p.slopes) return false;
	const float4 *MS = p.smom + sn + 2 * ((size_t)cy * p.sWp + cx), *TS = p.tmom + tn + 2 * ((size_t)y * p.tWp + x);
#pragma unroll
	for (int j = 0; j < 2; j++) {
		const float4 f0 = f4_sub(__ldg(MS + j), __ldg(TS + j));
		add(f0, false);
		if (Kind<KIND>::grad) {
			add(f4_sub(f4_sub(__ldg(MS + 2 + j), __ldg(TS + 2 + j)), f0), true);
			add(f4_sub(f4_sub(__ldg(MS + 2 * p.sWp + j), __ldg(TS + 2 * p.tWp + j)), f0), true);
		}
	}
	return exceeds();
}

// The tables' tap weights, one factor per axis: w and w f (f_1 along x, f_2
// along y; patch_factors in patchmatch.cu).
struct PmFactors {
	int px, py, rx, ry;
	float wx[NLI_MAX_PATCH], wy[NLI_MAX_PATCH], fx[NLI_MAX_PATCH], fy[NLI_MAX_PATCH];
};

// Rows after which an evaluation is tested for early termination (counted
// from 0): every term is non-negative, so once the rows summed so far reach
// the current distance for every candidate of a round, the rest of the round
// is skipped (exact).  9 x 9 L2 combined: after 4 of 10 rows.  Over the
// 512 x 512 NL-Poisson process() without the lower bound that stops 57.5 %
// of the candidates and was 1.6 % faster than a test at half the window
// (65 % stopped); two tests (rows 5 and 7, or 3 and 5 and 7) cost more than
// they save.
template <int P, int G>
__device__ __forceinline__ constexpr int check_row()
{
	return (P + G) / 2 - 2;
}

// A warp's counts in shared memory (kept by lane 0): candidates evaluated, of
// these at their point's distance by the early test, points that propagation
// improved; registers are what limits the warps per SM.
struct PmCount {
	unsigned evals, partial, improved, pad;
};

// The first pixel of the window around target (x, y), in the padded target.
__device__ __forceinline__ int tgt_window(const PmArgs &p, int x, int y) { return (y - p.ry) * p.tWp + (x - p.rx); }

// One round: this lane's part (column c of sub-warp sw) of candidate `cand`
// (x | y << 15) against the target whose window starts at t (tgt_window: target
// sides have no limit, so no packed position holds them).  Lanes with c == 0 return
// their sub-warp's distance, or infinity when every active candidate of the
// warp had reached its `bound` by the early test.  count->partial takes the
// active candidates that had reached `start` by then.
// P > 0: square P x P patch known at compile time (rows unrolled); P == 0:
// sizes from the arguments.
template <int KIND, int C, int P>
__device__ __forceinline__ float eval_round(const PmArgs &p, const float *s_w, unsigned cand, int t, int sw, int c,
                                            bool active, float bound, float start, PmCount *count)
{
	constexpr bool G = Kind<KIND>::grad;
	const int L = P ? P + G : p.L;
	const int K = P ? 32 / (P + G) : p.K;
	const int rows = P ? P + G : p.rows;
	const int px = P ? P : p.rx + p.ex;
	const int py = P ? P : p.ry + p.ey;
	const bool tapcol = c < px;
	const float *W = s_w + c;
	const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
	// this lane's pixel of the next row to load (sides below 32768: 31 bits)
	int so = ((int)((cand >> 15) & 0x7fffu) - p.ry) * p.sWp + ((int)(cand & 0x7fffu) - p.rx) + c;
	int to = t + c;
	const int s_n = p.sWp * (p.sH + 1), t_n = p.tWp * (p.tH + 1);
	auto load_s = [&](float4 &v) {
		// the lanes left over hold no column of a window
		if (sw < K && nli_in_bounds(so, s_n, kSitePmSource)) v = __ldg(p.src + so);
		so += p.sWp;
	};
	auto load_t = [&](float4 &v) {
		if (sw < K && nli_in_bounds(to, t_n, kSitePmWindow)) v = __ldg(p.tgt + to);
		to += p.tWp;
	};
	// source rows in flight (fewer for 4 channels: registers); the target's
	// window is the warp's own and in L1 after the first candidate
	constexpr int PF = C == 4 ? 1 : 2;
	float4 v[PF], u = zero;
#pragma unroll
	for (int r = 0; r < PF; r++) {
		v[r] = zero;
		if (r < rows) load_s(v[r]);
	}
	load_t(u);
	float4 dp = zero;
	float wp = 0.f;
	Acc A = {0.f, 0.f, 0.f, 0.f};
	bool stop = false;
	auto row = [&](int r, float4 &vr) {
		const float4 d = subc<C>(vr, u);
		const bool tap = tapcol && r < py;
		const float w = tap ? W[r * px] : 0.f;
		if (r + PF < rows) load_s(vr);
		if (r + 1 < rows) load_t(u);
		row_terms<KIND, C>(d, dp, w, wp, tap, G && tapcol && r > 0, A);
		dp = d;
		wp = w;
	};
	auto check = [&]() {
		const float part = subwarp_sum(combine<KIND>(A, p), c, L);
		const unsigned reached = __ballot_sync(kFull, active && c == 0 && part >= start);
		if (reached && (threadIdx.x & 31) == 0) count->partial += __popc(reached);
		return __all_sync(kFull, !active || c != 0 || part >= bound);
	};
	if constexpr (P > 0) {
#pragma unroll
		for (int r = 0; r < P + G; r++) {
			row(r, v[r % PF]);
			if (r == check_row<P, G>() && check()) {
				stop = true;
				break;
			}
		}
	} else {
#pragma unroll 1
		for (int r0 = 0; r0 < rows && !stop; r0 += PF) {
#pragma unroll
			for (int i = 0; i < PF; i++) {
				const int r = r0 + i;
				if (r >= rows) break;
				row(r, v[i]);
				if (r == rows / 2 && check()) {
					stop = true;
					break;
				}
			}
		}
	}
	if (stop) return __int_as_float(0x7f800000);
	return subwarp_sum(combine<KIND>(A, p), c, L);
}

// Evaluates the list's n entries (candidate x | y << 15 | group << 30), K at a
// time, and accepts each in order when strictly better than the match of
// the point it belongs to.  A lane holds its own point's state: group index
// g, target window twin (tgt_window), match (as the list's, without the
// group) and distance bd; lane g * lanes speaks for group g.  A candidate
// counts as partial against its point's distance of before the call, which
// does not depend on how points are grouped.
template <int KIND, int C, int P>
__device__ __forceinline__ void eval_list(const PmArgs &p, const float *s_w, const unsigned *list, int n, int g,
                                          int twin, unsigned &match, float &bd, PmCount *count)
{
	constexpr bool G = Kind<KIND>::grad;
	const int L = P ? P + G : p.L;
	const int K = P ? 32 / (P + G) : p.K;
	const int lane = threadIdx.x & 31;
	const int sw = lane / L, c = lane - sw * L;
	const float bd0 = bd;
#pragma unroll 1
	for (int b = 0; b < n; b += K) {
		const int idx = b + sw;
		const bool active = sw < K && idx < n;
		// idle lanes repeat the round's first entry; nothing reads their sums
		const unsigned e = list[active ? idx : b];
		const int speaker = (int)(e >> 30) * p.group.lanes;
		const int t = __shfl_sync(kFull, twin, speaker);
		const float bound = __shfl_sync(kFull, bd, speaker), start = __shfl_sync(kFull, bd0, speaker);
		const float sum = eval_round<KIND, C, P>(p, s_w, e, t, sw, c, active, bound, start, count);
		const int in_round = min(K, n - b);
#pragma unroll 1
		for (int s = 0; s < in_round; s++) {
			const float ds = __shfl_sync(kFull, sum, s * L);
			const unsigned es = __shfl_sync(kFull, e, s * L);
			if ((int)(es >> 30) == g && ds < bd) {
				bd = ds;
				match = es & 0x3fffffffu;
			}
		}
	}
}

// The one-point variants: evaluates the n candidates held one per lane (packed
// x | y << 16, lane i holds candidate i) in steps of K and accepts each in
// order when strictly better than the current match.  All lanes return the
// same best / bd.  kPmStaged: the step's source windows are copied into the
// warp's slots first (one tensor copy per candidate) and the rows are read
// from there, the target rows from s_t.  kPmRegs: the source rows are plain
// loads and the target rows come from tw (registers).
template <int KIND, int C, int P, int V>
__device__ __forceinline__ void eval_candidates(const PmArgs &p, const float *s_w, const float4 *s_t, int mycand,
                                                int n, int2 &best, float &bd, unsigned &partial, TmaState *ts,
                                                const float4 *tw)
{
	static_assert(P > 0 && V != kPmGrouped, "compiled for fixed patch sizes");
	constexpr bool TMA = V == kPmStaged;
	constexpr bool G = Kind<KIND>::grad;
	constexpr int PF = (C == 4) ? 1 : 2;
	constexpr int L = P + G, K = 32 / L, rows = P + G;
	if (TMA && ts->map == nullptr) return;  // this warp's staging gave up (timeout flagged)
	const int lane = threadIdx.x & 31;
	const int sw = lane / L, c = lane - sw * L;
	const bool tapcol = c < P;
	const size_t sWp = (size_t)p.sWp;
	const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
	const float bd0 = bd;  // what a partial candidate is counted against, as in eval_list
#pragma unroll 1
	for (int b = 0; b < n; b += K) {
		const int idx = b + sw;
		const bool active = sw < K && idx < n;
		const bool act_col = active && tapcol;
		const int cand = __shfl_sync(kFull, mycand, active ? idx : 0);
		const int cx = cand & 0xffff, cy = cand >> 16;
		const float4 *S = p.src + (size_t)(cy - p.ry) * sWp + (cx - p.rx) + c;
		// row r of this lane's column of the candidate's window (a checked
		// build tests the index against the padded source)
		const long long s_base = (long long)(cy - p.ry) * (long long)sWp + (cx - p.rx) + c;
		const long long s_n = (long long)sWp * (p.sH + 1);
		auto ldrow = [&](int r) -> float4 {
			return nli_in_bounds(s_base + (long long)r * (long long)sWp, s_n, kSitePmSource) ? __ldg(S + (size_t)r * sWp)
			                                                                                 : zero;
		};
		const float4 *T = s_t + c;
		const float *Wt = s_w + c;
		const float4 *Sl = nullptr;  // this lane's column of its candidate's staged window
		if constexpr (TMA) {
			const int nact = min(K, n - b);
			int cs[K];
#pragma unroll
			for (int s = 0; s < K; s++) cs[s] = __shfl_sync(kFull, mycand, min(b + s, 31));
			__syncwarp();
			if (lane == 0) {
				fence_proxy_async();
				mbar_expect_tx(ts->bar, (unsigned)(nact * rows * L * sizeof(float4)));
#pragma unroll
				for (int s = 0; s < K; s++)
					if (s < nact)
						tma_load_2d(ts->slots + s * ts->slot_stride, ts->map, 4 * ((cs[s] & 0xffff) - p.rx),
						            (cs[s] >> 16) - p.ry, ts->bar);
			}
			const bool landed = __all_sync(kFull, mbar_wait(ts->bar, ts->phase));
			if (!landed) {
				// the copies did not land in time: flag it, give them one more
				// bounded wait, and stop using this warp's slots
				if (lane == 0) atomicExch(ts->timeout, 1);
				mbar_wait(ts->bar, ts->phase);
				ts->map = nullptr;
				return;
			}
			ts->phase ^= 1u;
			Sl = ts->slots + (active ? sw : 0) * ts->slot_stride + c;
		}
		float4 v0 = (!TMA && active) ? ldrow(0) : zero;
		float4 v1 = (!TMA && PF == 2 && active) ? ldrow(1) : zero;
		float4 dp = zero;
		float wp = 0.f;
		Acc A = {0.f, 0.f, 0.f, 0.f};
		const float bound = bd;
		bool stop = false;
		auto row = [&](int r) {
			float4 v = v0;
			if (TMA) {
				v = active ? Sl[r * L] : zero;
			} else if (PF == 2) {
				v0 = v1;
				v1 = (active && r + 2 < rows) ? ldrow(r + 2) : zero;
			} else {
				v0 = (active && r + 1 < rows) ? ldrow(r + 1) : zero;
			}
			float4 t;
			if constexpr (V == kPmRegs)
				t = tw[r];
			else
				t = T[r * L];
			const float4 d = subc<C>(v, t);
			const bool tap = act_col && r < P;
			const float w = (C <= 3) ? t.w : (tap ? Wt[r * P] : 0.f);
			row_terms<KIND, C>(d, dp, w, wp, tap, G && act_col && r > 0, A);
			dp = d;
			wp = w;
		};
		auto check = [&]() {
			const float part = subwarp_sum(combine<KIND>(A, p), c, L);
			partial += __popc(__ballot_sync(kFull, active && c == 0 && part >= bd0));
			return __all_sync(kFull, !active || c != 0 || part >= bound);
		};
#pragma unroll
		for (int r = 0; r < rows; r++) {
			row(r);
			if (r == check_row<P, G>() && check()) {
				stop = true;
				break;
			}
		}
		if (stop) continue;
		const int in_step = min(K, n - b);
		const float sum = subwarp_sum(combine<KIND>(A, p), c, L);
#pragma unroll 1
		for (int s = 0; s < in_step; s++) {
			const float ds = __shfl_sync(kFull, sum, s * L);
			if (ds < bd) {
				bd = ds;
				const int q = __shfl_sync(kFull, mycand, b + s);
				best = make_int2(q & 0xffff, q >> 16);
			}
		}
	}
}

// Candidates proposed one per lane, in lane order: keeps the valid ones that
// differ from the current match and from every lower lane's candidate and
// moves them to lanes 0..n-1 (mycand), in order.  Returns n.
__device__ __forceinline__ int compact_candidates(bool valid, int packed, const int2 &best, int *s_list, int &mycand)
{
	const int lane = threadIdx.x & 31;
	const unsigned below = (1u << lane) - 1u;
	valid = valid && packed != (best.x | (best.y << 16));
	const unsigned vmask = __ballot_sync(kFull, valid);
	const unsigned same = __match_any_sync(kFull, valid ? packed : -1);
	const bool keep = valid && (same & vmask & below) == 0;
	const unsigned kmask = __ballot_sync(kFull, keep);
	if (keep) s_list[__popc(kmask & below)] = packed;
	__syncwarp();
	const int n = __popc(kmask);
	mycand = (lane < n) ? s_list[lane] : 0;
	__syncwarp();
	return n;
}

// Shared memory of the PatchMatch kernels: per-tap weights, then per warp a
// candidate list (32 ints).
struct PmSmem {
	float *w;
	int *list;
	float4 *t;      // staged path: the target window, rows x L float4
	float4 *slots;  // staged path: K windows per warp
	int slot_stride;
	uint64_t *bar;
};

// Staged path layout (float4 units, from a 128-byte aligned base): the
// weights, then per warp a region of the target window, K window slots, the
// candidate list and the mbarrier, every part starting on 128 bytes.
__host__ __device__ inline int pm_round8(int v) { return (v + 7) & ~7; }

__host__ __device__ inline int pm_tma_region(int rows, int L, int K)
{
	return pm_round8(pm_round8(rows * L) * (1 + K) + 8 + 1);
}

__host__ __device__ inline size_t pm_smem_bytes_tma(int taps, int rows, int L, int K, int warps)
{
	return 128 + sizeof(float4) * ((size_t)pm_round8(pm_weight_slots(taps)) + (size_t)warps * pm_tma_region(rows, L, K));
}

template <int V>
__device__ __forceinline__ PmSmem pm_smem(const DistArgs &a, const PmArgs &p)
{
	extern __shared__ float4 s_pm[];
	const int warp = threadIdx.x >> 5;
	PmSmem m;
	const int ws = pm_weight_slots(a.px * a.py);
	if (V != kPmStaged) {
		m.w = reinterpret_cast<float *>(s_pm);
		m.t = nullptr;
		m.list = reinterpret_cast<int *>(s_pm + ws) + warp * 36;
		m.slots = nullptr;
		m.slot_stride = 0;
		m.bar = nullptr;
	} else {
		float4 *base = reinterpret_cast<float4 *>((reinterpret_cast<uintptr_t>(s_pm) + 127) & ~(uintptr_t)127);
		const int win = pm_round8(p.rows * p.L);
		float4 *r = base + pm_round8(ws) + (size_t)warp * pm_tma_region(p.rows, p.L, p.K);
		m.w = reinterpret_cast<float *>(base);
		m.t = r;
		m.slots = r + win;
		m.slot_stride = win;
		m.list = reinterpret_cast<int *>(r + win * (1 + p.K));
		m.bar = reinterpret_cast<uint64_t *>(r + win * (1 + p.K) + 8);
	}
	return m;
}

// A target point's seed match (patch_match.cpp:341-381): the init field's
// where it lies in the source, otherwise redrawn uniformly up to `shots`
// times; (x, y) where !src_ok remains when the draws run out.
__device__ __forceinline__ int2 seed_match(const PmArgs &p, const uint2 key, int pix, const int2 *__restrict__ init)
{
	Rng rng(key, (uint32_t)pix, 0xffffffffu);
	int2 n = init ? init[pix] : make_int2(-1, -1);
	int tries = 0;
	while (!src_ok(p, n.x, n.y) && tries < p.shots) {
		n.x = rng.below(p.sW);
		n.y = rng.below(p.sH);
		tries++;
	}
	return n;
}

// One target point of the initial field (patch_match.cpp:329-381): its
// seed match and that match's distance.  Called by one whole warp; lane 0
// writes the results.
template <int KIND, int C, int P, int V>
__device__ __forceinline__ void pm_init_point(const PmArgs &p, const PmSmem &m, TmaState &ts, float4 *tw,
                                              const uint2 key, int pix, const int2 *__restrict__ init,
                                              int2 *__restrict__ nnf, float *__restrict__ dist, unsigned &evals,
                                              unsigned &partial)
{
	const int lane = threadIdx.x & 31;
	if (!nli_in_bounds(pix, (long long)p.tW * p.tH, kSitePmTarget)) return;
	const int x = pix % p.tW, y = pix / p.tW;
	const int2 n = seed_match(p, key, pix, init);
	float d = FLT_MAX;
	int2 best = make_int2(-1, -1);
	if (src_ok(p, n.x, n.y) && tgt_patch_inside(p, x, y)) {
		if constexpr (V == kPmRegs)
			load_window_regs<KIND, C, P>(p, m.w, x, y, tw);
		else
			load_window<KIND, C, P>(p, m.w, x, y, m.t);
		eval_candidates<KIND, C, P, V>(p, m.w, m.t, n.x | (n.y << 16), 1, best, d, partial, &ts, tw);
		evals++;
		__syncwarp();
	}
	if (lane == 0) {
		nnf[pix] = best;
		dist[pix] = d;
	}
}

template <int KIND, int C, int P, int V>
__global__ void __launch_bounds__(pm_threads(V), 1) k_pm_init(DistArgs a, PmArgs p, const int2 *__restrict__ init,
                                                      int2 *__restrict__ nnf, float *__restrict__ dist,
                                                      unsigned long long *counter,
                                                      const __grid_constant__ CUtensorMap tmap, int *timeout)
{
	const int lane = threadIdx.x & 31;
	const PmSmem m = pm_smem<V>(a, p);
	TmaState ts = {&tmap, m.slots, m.slot_stride, m.bar, 0u, timeout};
	if (V == kPmStaged && lane == 0) mbar_init(m.bar, 1);
	float4 tw[(V == kPmRegs) ? P + 1 : 1];
	load_weights(a, m.w);
	const uint2 key = pm_key(p);
	unsigned evals = 0, partial = 0;
	pm_for_each(p.nt, p.queue, p.tile, [&](int wi) {
		pm_init_point<KIND, C, P, V>(p, m, ts, tw, key, p.tlist[wi], init, nnf, dist, evals, partial);
	});
	if (lane == 0 && evals) {
		atomicAdd(counter, (unsigned long long)evals);
		if (partial) atomicAdd(counter + 1, (unsigned long long)partial);
	}
}

// What one sweep reads and writes.
struct PmIo {
	const int2 *nnf_in;
	const float *dist_in;
	const uint8_t *hist_in;
	int2 *nnf_out;
	float *dist_out;
	uint8_t *hist_out;
};

// A call's field, distances and change histories (seen_before), each twice:
// sweep s reads x and writes y when s is even, the other way round when odd.
struct PmFields {
	int2 *nnf_x, *nnf_y;
	float *dist_x, *dist_y;
	uint8_t *hist_x, *hist_y;
	PmIo io(int sweep) const
	{
		return (sweep % 2) == 0 ? PmIo{nnf_x, dist_x, hist_x, nnf_y, dist_y, hist_y}
		                        : PmIo{nnf_y, dist_y, hist_y, nnf_x, dist_x, hist_x};
	}
};

// Whether a neighbour's proposal needs no evaluation because the same
// proposal was already tried for this point in this call.  Bit i of a
// point's history says whether sweep s - 1 - i changed its match.  The
// neighbours at distance 1 are asked every sweep, those at the jump distance
// every fourth sweep with the same distance (jump_for); when the neighbour's
// match has not changed since, its proposal is the one of that earlier sweep.
// It was then evaluated, or ruled out by the lower bound, against a distance
// that has only fallen since, so it cannot be strictly better now: the field
// and distances are those of evaluating it again.
// On the 512 x 512 NL-Poisson process() this takes the evaluations from 1.09
// to 0.69 x 10^9 and the run from 724 to 657 ms; a first call from random
// matches on 512 x 512 goes from 1706 to 1567 us.
__device__ __forceinline__ bool seen_before(unsigned hist, int sweep, bool at_jump)
{
	return at_jump ? sweep >= 4 && (hist & 15u) == 0u : sweep >= 1 && (hist & 1u) == 0u;
}

// Whether (cx, cy) is a usable source centre that the lower bound does not
// rule out for target (x, y).  Usable centres are nearly all of those
// proposed, so the bound's loads are issued beside the mask's.
template <int KIND, int C>
__device__ __forceinline__ bool src_takes(const PmArgs &p, int x, int y, int cx, int cy, float bd)
{
	if (!src_inside(p, cx, cy)) return false;
	const bool usable = src_masked(p, cx, cy);
	const bool rejected = p.smom && bound_rejects<KIND, C>(p, x, y, cx, cy, bd);
	return usable && !rejected;
}

// Proposal k (0-7) of a point's propagation step: the match of neighbour
// k & 3 (left, right, up, down) at distance 1 (k < 4) or at the jump distance,
// shifted back by the neighbour's offset.  False when there is none to
// evaluate.
template <int KIND, int C>
__device__ __forceinline__ bool propagated(const PmArgs &p, int x, int y, int k, int sweep, int jump,
                                           const PmIo &io, float bd, int &cx, int &cy)
{
	const int s = (k < 4) ? 1 : jump, side = k & 3;
	const int nx = x + ((side == 0) ? -s : (side == 1) ? s : 0);
	const int ny = y + ((side == 2) ? -s : (side == 3) ? s : 0);
	// the loads of a step are issued together (a point is a chain of them):
	// outside the image, where nothing is proposed, they read the point itself
	const bool in = (unsigned)nx < (unsigned)p.tW && (unsigned)ny < (unsigned)p.tH;
	const int at = in ? ny * p.tW + nx : y * p.tW + x;
	if (!nli_in_bounds(at, (long long)p.tW * p.tH, kSitePmField)) return false;
	const uint8_t target = p.tmask[at];
	const int2 q = io.nnf_in[at];
	const unsigned hist = sweep ? io.hist_in[at] : 0u;
	if (!in || !target || q.x < 0 || seen_before(hist, sweep, k >= 4)) return false;
	cx = q.x + (x - nx);
	cy = q.y + (y - ny);
	return src_takes<KIND, C>(p, x, y, cx, cy, bd);
}

// Proposal k of a point's random search around its match (bx, by): up to
// `shots` draws in window max_window >> k from the proposal's own stream, the
// first that lands in the source.  False when there is none to evaluate.
// One Philox block holds two draws; which draw of its stream a proposal ends
// on depends on the draws alone.
template <int KIND, int C>
__device__ __forceinline__ bool drawn(const PmArgs &p, const uint2 key, int pix, int x, int y, int bx, int by, int k,
                                      int sweep, float bd, int &cx, int &cy, int &max_shot)
{
	const int w = p.max_window >> k;
	const int x_min = max(bx - w, 0), y_min = max(by - w, 0);
	const uint32_t nx = (uint32_t)(min(bx + w + 1, p.sW) - x_min), ny = (uint32_t)(min(by + w + 1, p.sH) - y_min);
#pragma unroll 1
	for (int t = 0; t < p.shots; t += 2) {
		const uint4 u = Rng::block_of(key, (uint32_t)pix, (uint32_t)sweep, (uint32_t)k, (uint32_t)t >> 1);
		cx = x_min + (int)__umulhi(u.x, nx);
		cy = y_min + (int)__umulhi(u.y, ny);
		bool ok = src_ok(p, cx, cy);
		int shot = t;
		if (!ok && t + 1 < p.shots) {
			cx = x_min + (int)__umulhi(u.z, nx);
			cy = y_min + (int)__umulhi(u.w, ny);
			ok = src_ok(p, cx, cy);
			shot = t + 1;
		}
		if (ok) {
			max_shot = max(max_shot, shot);
			return !(p.smom && bound_rejects<KIND, C>(p, x, y, cx, cy, bd));
		}
	}
	return false;
}

// The one-point variants' target point of a sweep: propagation from the
// previous sweep's field, then random search around the best match.  Called
// by one whole warp; lane 0 writes the results.
template <int KIND, int C, int P, int V>
__device__ __forceinline__ void pm_sweep_point(const PmArgs &p, const PmSmem &m, TmaState &ts, float4 *tw,
                                               const uint2 key, int windows, int pix, int sweep, int jump,
                                               const PmIo &io,
                                               unsigned &evals, unsigned &partial, unsigned &improved, int &max_shot)
{
	const int lane = threadIdx.x & 31;
	if (!nli_in_bounds(pix, (long long)p.tW * p.tH, kSitePmTarget)) return;
	const int x = pix % p.tW, y = pix / p.tW;
	int2 best = io.nnf_in[pix];
	float bd = io.dist_in[pix];
	const float bd_in = bd;
	const unsigned hist = sweep ? io.hist_in[pix] : 0u;
	if (tgt_patch_inside(p, x, y)) {
		if constexpr (V == kPmRegs)
			load_window_regs<KIND, C, P>(p, m.w, x, y, tw);
		else
			load_window<KIND, C, P>(p, m.w, x, y, m.t);
		int cx = 0, cy = 0;
		bool valid = lane < (jump > 1 ? 8 : 4) &&
		             propagated<KIND, C>(p, x, y, lane, sweep, jump, io, bd, cx, cy);
		int mycand;
		int n = compact_candidates(valid, cx | (cy << 16), best, m.list, mycand);
		evals += n;
		const float bd_before = bd;
		eval_candidates<KIND, C, P, V>(p, m.w, m.t, mycand, n, best, bd, partial, &ts, tw);
		if (bd < bd_before) improved++;
		cx = cy = 0;
		valid = lane < windows &&
		        drawn<KIND, C>(p, key, pix, x, y, best.x, best.y, lane, sweep, bd, cx, cy, max_shot);
		n = compact_candidates(valid, cx | (cy << 16), best, m.list, mycand);
		evals += n;
		eval_candidates<KIND, C, P, V>(p, m.w, m.t, mycand, n, best, bd, partial, &ts, tw);
		__syncwarp();
	} else {
		best = make_int2(-1, -1);
		bd = FLT_MAX;
	}
	if (lane == 0) {
		io.nnf_out[pix] = best;
		io.dist_out[pix] = bd;
		// a match changes only together with a strictly smaller distance
		io.hist_out[pix] = (uint8_t)((hist << 1) | (bd < bd_in ? 1u : 0u));
	}
}

// ------------------------------------------------------ groups of points
// A lane's place in its warp's group: point g, lane k of that point's.
struct PmLane {
	int g, k;
};

__device__ __forceinline__ PmLane pm_lane(const PmGroup &group)
{
	const int lane = threadIdx.x & 31;
	const int g = lane / group.lanes;
	return {g, lane - g * group.lanes};
}

constexpr unsigned kNoMatch = 0xffffffffu;

// The counts behind a warp's list.
__device__ __forceinline__ PmCount *pm_count(unsigned *list) { return reinterpret_cast<PmCount *>(list + 32); }

__device__ __forceinline__ void pm_count_clear(unsigned *list)
{
	if ((threadIdx.x & 31) < 4) list[32 + (threadIdx.x & 31)] = 0u;
	__syncwarp();
}

// The warp's list of proposals (one per lane at most, packed x | y << 15 with
// the group above): those that are valid, differ from their point's match and
// from every lower lane's for the same point.  Returns their number.
__device__ __forceinline__ int list_proposals(bool valid, unsigned packed, unsigned match, int g, unsigned *list,
                                              bool counts = true)
{
	const int lane = threadIdx.x & 31;
	const unsigned below = (1u << lane) - 1u;
	valid = valid && packed != match;
	const unsigned entry = packed | ((unsigned)g << 30);
	const unsigned vmask = __ballot_sync(kFull, valid);
	if (vmask == 0) return 0;
	const unsigned same = __match_any_sync(kFull, valid ? entry : kNoMatch);
	const bool keep = valid && (same & vmask & below) == 0;
	const unsigned kmask = __ballot_sync(kFull, keep);
	__syncwarp();
	if (keep) list[__popc(kmask & below)] = entry;
	if (lane == 0 && counts) pm_count(list)->evals += __popc(kmask);
	__syncwarp();
	return __popc(kmask);
}

// Points [first, first + group.points) of the initial field.
template <int KIND, int C, int P>
__device__ __forceinline__ void pm_init_group(const PmArgs &p, const float *s_w, unsigned *list, const PmLane at,
                                              const uint2 key, int first, const int2 *__restrict__ init,
                                              int2 *__restrict__ nnf, float *__restrict__ dist)
{
	PmCount *count = pm_count(list);
	bool has = at.g < p.group.points && first + at.g < p.nt;
	const int pix = has ? p.tlist[first + at.g] : 0;
	has = has && nli_in_bounds(pix, (long long)p.tW * p.tH, kSitePmTarget);
	const int x = pix % p.tW, y = pix / p.tW;
	int2 n = make_int2(0, 0);
	bool valid = false;
	if (has) {
		n = seed_match(p, key, pix, init);
		valid = src_ok(p, n.x, n.y) && tgt_patch_inside(p, x, y);
	}
	unsigned match = kNoMatch;
	float d = FLT_MAX;
	const int listed = list_proposals(valid && at.k == 0, (unsigned)n.x | ((unsigned)n.y << 15), match, at.g, list);
	eval_list<KIND, C, P>(p, s_w, list, listed, at.g, tgt_window(p, x, y), match, d, count);
	if (has && at.k == 0) {
		nnf[pix] = match == kNoMatch ? make_int2(-1, -1) : make_int2(match & 0x7fffu, match >> 15);
		dist[pix] = d;
	}
}

// Points [first, first + group.points) of a sweep: propagation from the
// previous sweep's field, then random search around each point's match.
template <int KIND, int C, int P>
__device__ __forceinline__ void pm_sweep_group(const PmArgs &p, const float *s_w, unsigned *list, const PmLane at,
                                               const uint2 key, int windows, int first, int sweep, int jump,
                                               const PmIo &io,
                                               int &max_shot)
{
	PmCount *count = pm_count(list);
	bool has = at.g < p.group.points && first + at.g < p.nt;
	const int pix = has ? p.tlist[first + at.g] : 0;
	has = has && nli_in_bounds(pix, (long long)p.tW * p.tH, kSitePmTarget);
	const int x = pix % p.tW, y = pix / p.tW;
	const int twin = tgt_window(p, x, y);
	const bool inside = has && tgt_patch_inside(p, x, y);
	unsigned match = kNoMatch;
	float bd = FLT_MAX;
	if (inside) {
		const int2 q = io.nnf_in[pix];
		if (q.x >= 0) match = (unsigned)q.x | ((unsigned)q.y << 15);
		bd = io.dist_in[pix];
	}
	const float bd_in = bd;
	int cx = 0, cy = 0;
	bool valid = inside && at.k < (jump > 1 ? 8 : 4) &&
	             propagated<KIND, C>(p, x, y, at.k, sweep, jump, io, bd, cx, cy);
	int n = list_proposals(valid, (unsigned)cx | ((unsigned)cy << 15), match, at.g, list);
	if (n) {
		eval_list<KIND, C, P>(p, s_w, list, n, at.g, twin, match, bd, count);
		const unsigned better = __ballot_sync(kFull, at.k == 0 && bd < bd_in);
		if (better && at.g == 0 && at.k == 0) count->improved += __popc(better);
	}
	const int bx = match == kNoMatch ? -1 : (int)(match & 0x7fffu), by = match == kNoMatch ? -1 : (int)(match >> 15);
	cx = cy = 0;
	valid = inside && at.k < windows &&
	        drawn<KIND, C>(p, key, pix, x, y, bx, by, at.k, sweep, bd, cx, cy, max_shot);
	n = list_proposals(valid, (unsigned)cx | ((unsigned)cy << 15), match, at.g, list);
	eval_list<KIND, C, P>(p, s_w, list, n, at.g, twin, match, bd, count);
	if (has && at.k == 0) {
		io.nnf_out[pix] = match == kNoMatch ? make_int2(-1, -1) : make_int2(match & 0x7fffu, match >> 15);
		io.dist_out[pix] = bd;
		// a match changes only together with a strictly smaller distance
		const unsigned hist = sweep ? io.hist_in[pix] : 0u;
		io.hist_out[pix] = (uint8_t)((hist << 1) | (inside && bd < io.dist_in[pix] ? 1u : 0u));
	}
}

// ------------------------------------------------- warps sharing a point
// Small calls: a block of NW warps takes one point at a time.  Such a sweep lasts
// as long as one point's chain of instructions (about 2900 in a first call,
// half of them in rounds), whatever the memory does, so the chain is cut:
// warp 0 proposes by propagation while the others already draw around the match
// as it is (the draws are made again where propagation improves it), a window's
// draws are tried by several lanes at once, and each warp evaluates its share of a
// step's candidates.  They are then accepted in the list's order, so the field
// is the one a single warp finds.  A sweep of 750 points (64 x 48, 9 x 9 patch)
// takes 14.3 us instead of 18.5, the call 252 us instead of 297; the coarse
// sweeps of a run at 256 x 256 (255 points) 13 us instead of 18.
// Blocks of NW warps per SM that the team kernels' registers are held to (80 a
// thread, where the 9 x 9 ones spill 16 bytes; at 64 they spill more and a sweep of 2
// warps a point is 5 % slower, at 128 too few points run at once: 20 us instead of 14
// for 750 points).
constexpr int team_blocks(int NW) { return 24 / NW; }

// Warps that share a point in a call of nt points; 1: points are grouped by
// warp.  A team is worth it while all its blocks run at once.  On 152 SMs,
// with limits of (6, 12), (8, 16), (10, 16) and (6, 24) points per SM for 4
// and 2 warps: a whole run at 256 x 256 takes 40.0, 40.5, 41.0 and 41.0 ms
// (43.2 without teams), one on 152 x 97 RGB-D 17.05, 17.2, 17.2 and 17.8 (17.05).
inline int pm_team(long long nt, int num_sms)
{
	return nt <= (long long)team_blocks(4) * num_sms ? 4 : nt <= (long long)team_blocks(2) * num_sms ? 2 : 1;
}

constexpr unsigned kNoProposal = 0xfffffffeu;

struct PmTeam {
	unsigned prop[8];    // propagation's proposals
	unsigned draw[32];   // random search's, by window
	int shot[32];        // which draw each was
	float dist[32];      // the step's distances
};

// Draws of windows first, first + stride, ... by one warp, lanes / window
// each: the first draw of a window's stream that lands in the source, tested by
// the bound, into team->draw and team->shot.
template <int KIND, int C>
__device__ __forceinline__ void team_draws(const PmArgs &p, const uint2 key, int pix, int x, int y, unsigned match,
                                           float bd, int windows, int sweep, int first, int stride, PmTeam *team)
{
	const int lane = threadIdx.x & 31;
	const int bx = match == kNoMatch ? -1 : (int)(match & 0x7fffu), by = match == kNoMatch ? -1 : (int)(match >> 15);
	const int mine = (windows - first + stride - 1) / stride;  // this warp's windows
	if (mine <= 0) return;
	const int per = 32 / mine;
	const int j = lane / per, sub = lane - j * per, k = first + stride * j;
	const bool has = j < mine;
	const unsigned group = has ? ((per == 32 ? kFull : (1u << per) - 1u) << (j * per)) : 0u;
	const int w = has ? p.max_window >> k : 0;  // (k runs past 31 in the lanes left over)
	const int x_min = max(bx - w, 0), y_min = max(by - w, 0);
	const uint32_t nx = (uint32_t)(min(bx + w + 1, p.sW) - x_min), ny = (uint32_t)(min(by + w + 1, p.sH) - y_min);
	bool found = !has;
	int cx = 0, cy = 0, shot = -1;
#pragma unroll 1
	for (int t0 = 0; t0 < p.shots; t0 += per) {
		const int t = t0 + sub;
		int qx = 0, qy = 0;
		bool ok = false;
		if (!found && t < p.shots) {
			const uint4 u = Rng::block_of(key, (uint32_t)pix, (uint32_t)sweep, (uint32_t)k, (uint32_t)t >> 1);
			qx = x_min + (int)__umulhi((t & 1) ? u.z : u.x, nx);
			qy = y_min + (int)__umulhi((t & 1) ? u.w : u.y, ny);
			ok = src_ok(p, qx, qy);
		}
		const unsigned hit = __ballot_sync(kFull, ok) & group;
		const int from = hit ? __ffs(hit) - 1 : lane;
		qx = __shfl_sync(kFull, qx, from);
		qy = __shfl_sync(kFull, qy, from);
		if (hit && !found) {
			cx = qx;
			cy = qy;
			shot = t0 + from - j * per;
			found = true;
		}
		if (__all_sync(kFull, found)) break;
	}
	const bool keep = has && shot >= 0 && !(p.smom && bound_rejects<KIND, C>(p, x, y, cx, cy, bd));
	if (has && sub == 0) {
		team->draw[k] = keep ? (unsigned)cx | ((unsigned)cy << 15) : kNoProposal;
		team->shot[k] = shot;
	}
}

// A step's proposals (in every warp's lanes alike) evaluated by the block's warps
// together and accepted in order.  `first`: the warp that counts.
template <int KIND, int C, int P, int NW>
__device__ __forceinline__ void team_step(const PmArgs &p, const float *s_w, unsigned *list, PmTeam *team, bool valid,
                                          unsigned packed, int twin, unsigned &match, float &bd)
{
	constexpr bool G = Kind<KIND>::grad;
	const int L = P ? P + G : p.L;
	const int K = P ? 32 / (P + G) : p.K;
	const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
	const int sw = lane / L, c = lane - sw * L;
	const int n = list_proposals(valid, packed, match, 0, list, wid == 0);
	if (n == 0) return;
	for (int b = wid * K; b < n; b += NW * K) {
		const int idx = b + sw;
		const bool active = sw < K && idx < n;
		const float d = eval_round<KIND, C, P>(p, s_w, list[active ? idx : b], twin, sw, c, active, bd, bd, pm_count(list));
		if (active && c == 0) team->dist[idx] = d;
	}
	__syncthreads();
	for (int i = 0; i < n; i++) {
		const float d = team->dist[i];
		if (d < bd) {
			bd = d;
			match = list[i];
		}
	}
	__syncthreads();
}

// One point of a sweep by the whole block.
template <int KIND, int C, int P, int NW>
__device__ __forceinline__ void pm_sweep_team(const PmArgs &p, const float *s_w, unsigned *list, PmTeam *team,
                                              const uint2 key, int windows, int pix, int sweep, int jump, const PmIo &io,
                                              int &max_shot)
{
	if (!nli_in_bounds(pix, (long long)p.tW * p.tH, kSitePmTarget)) return;
	const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
	const int x = pix % p.tW, y = pix / p.tW;
	const int twin = tgt_window(p, x, y);
	unsigned match = kNoMatch;
	float bd = FLT_MAX;
	const bool inside = tgt_patch_inside(p, x, y);
	if (inside) {
		const int2 q = io.nnf_in[pix];
		bd = io.dist_in[pix];
		if (q.x >= 0) match = (unsigned)q.x | ((unsigned)q.y << 15);
		const unsigned before = match;
		if (wid == 0) {
			int cx = 0, cy = 0;
			const bool valid = lane < (jump > 1 ? 8 : 4) && propagated<KIND, C>(p, x, y, lane, sweep, jump, io, bd, cx, cy);
			if (lane < 8) team->prop[lane] = valid ? (unsigned)cx | ((unsigned)cy << 15) : kNoProposal;
		} else {
			team_draws<KIND, C>(p, key, pix, x, y, match, bd, windows, sweep, wid - 1, NW - 1, team);
		}
		__syncthreads();
		unsigned packed = lane < 8 ? team->prop[lane] : kNoProposal;
		team_step<KIND, C, P, NW>(p, s_w, list, team, packed != kNoProposal, packed, twin, match, bd);
		if (match != before) {
			if (wid == 0 && lane == 0) pm_count(list)->improved++;
			team_draws<KIND, C>(p, key, pix, x, y, match, bd, windows, sweep, wid, NW, team);
			__syncthreads();
		}
		packed = lane < windows ? team->draw[lane] : kNoProposal;
		if (wid == 0 && lane < windows) max_shot = max(max_shot, team->shot[lane]);
		team_step<KIND, C, P, NW>(p, s_w, list, team, packed != kNoProposal, packed, twin, match, bd);
	}
	if (threadIdx.x == 0) {
		io.nnf_out[pix] = match == kNoMatch ? make_int2(-1, -1) : make_int2(match & 0x7fffu, match >> 15);
		io.dist_out[pix] = bd;
		// a match changes only together with a strictly smaller distance
		const unsigned hist = sweep ? io.hist_in[pix] : 0u;
		io.hist_out[pix] = (uint8_t)((hist << 1) | (inside && bd < io.dist_in[pix] ? 1u : 0u));
	}
}

// Adds a warp's candidate counts to `counter` (and to `image`'s, if given).
__device__ __forceinline__ void pm_count_add(unsigned *list, unsigned long long *counter, unsigned long long *image)
{
	const PmCount *c = pm_count(list);
	if ((threadIdx.x & 31) == 0 && (c->evals || c->partial)) {
		if (c->evals) atomicAdd(counter, (unsigned long long)c->evals);
		if (c->partial) atomicAdd(counter + 1, (unsigned long long)c->partial);
		if (image) {
			if (c->evals) atomicAdd(image, (unsigned long long)c->evals);
			if (c->partial) atomicAdd(image + 1, (unsigned long long)c->partial);
		}
	}
	__syncwarp();
}

template <int KIND, int C, int P>
__global__ void __launch_bounds__(pm_threads(kPmGrouped), 1)
    k_pm_init_grouped(DistArgs a, PmArgs p, const int2 *__restrict__ init, int2 *__restrict__ nnf,
                      float *__restrict__ dist, unsigned long long *counter)
{
	const PmSmem m = pm_smem<kPmGrouped>(a, p);
	next_launch_may_start();
	load_weights(a, m.w);
	previous_launch_done();
	const uint2 key = pm_key(p);
	const PmLane at = pm_lane(p.group);
	unsigned *list = reinterpret_cast<unsigned *>(m.list);
	pm_count_clear(list);
	const int groups = (p.nt + p.group.points - 1) / p.group.points;
	pm_for_each(groups, p.queue, p.tile, [&](int i) {
		pm_init_group<KIND, C, P>(p, m.w, list, at, key, i * p.group.points, init, nnf, dist);
	});
	pm_count_add(list, counter, nullptr);
}

// metric_prop (may be NULL): this sweep's count of target points that the
// propagation step improved; metric_shots (may be NULL): the largest index
// of a first accepted random draw (patch_match.cpp:452-456, 481-485).
template <int KIND, int C, int P>
__global__ void __launch_bounds__(pm_threads(kPmGrouped), 1)
    k_pm_sweep_grouped(DistArgs a, PmArgs p, int sweep, int jump, PmIo io, unsigned long long *counter, unsigned long long *metric_prop, int *metric_shots)
{
	const int lane = threadIdx.x & 31;
	const PmSmem m = pm_smem<kPmGrouped>(a, p);
	next_launch_may_start();
	load_weights(a, m.w);
	previous_launch_done();
	const uint2 key = pm_key(p);
	const PmLane at = pm_lane(p.group);
	unsigned *list = reinterpret_cast<unsigned *>(m.list);
	pm_count_clear(list);
	int max_shot = -1;
	// number of random-search windows: max_window, max_window / 2, ..., 1
	const int windows = 32 - __clz(p.max_window);
	const int groups = (p.nt + p.group.points - 1) / p.group.points;
	pm_for_each(groups, p.queue ? p.queue + 1 + sweep : nullptr, p.tile, [&](int i) {
		pm_sweep_group<KIND, C, P>(p, m.w, list, at, key, windows, i * p.group.points, sweep, jump, io, max_shot);
	});
	pm_count_add(list, counter, nullptr);
	if (metric_prop && lane == 0 && pm_count(list)->improved)
		atomicAdd(metric_prop, (unsigned long long)pm_count(list)->improved);
	if (metric_shots) {
		max_shot = __reduce_max_sync(kFull, max_shot);
		if (lane == 0 && max_shot >= 0) atomicMax(metric_shots, max_shot);
	}
}

// metric_prop (may be NULL): this sweep's count of target points that the
// propagation step improved; metric_shots (may be NULL): the largest index
// of a first accepted random draw (patch_match.cpp:452-456, 481-485).
template <int KIND, int C, int P, int V>
__global__ void __launch_bounds__(pm_threads(V), 1) k_pm_sweep(DistArgs a, PmArgs p, int sweep, int jump,
                                                       PmIo io, unsigned long long *counter, unsigned long long *metric_prop,
                                                       int *metric_shots, const __grid_constant__ CUtensorMap tmap,
                                                       int *timeout)
{
	const int lane = threadIdx.x & 31;
	const PmSmem m = pm_smem<V>(a, p);
	TmaState ts = {&tmap, m.slots, m.slot_stride, m.bar, 0u, timeout};
	if (V == kPmStaged && lane == 0) mbar_init(m.bar, 1);
	float4 tw[(V == kPmRegs) ? P + 1 : 1];
	load_weights(a, m.w);
	const uint2 key = pm_key(p);
	unsigned evals = 0, partial = 0, improved = 0;
	int max_shot = -1;
	// number of random-search windows: max_window, max_window / 2, ..., 1
	const int windows = 32 - __clz(p.max_window);
	pm_for_each(p.nt, p.queue ? p.queue + 1 + sweep : nullptr, p.tile, [&](int wi) {
		pm_sweep_point<KIND, C, P, V>(p, m, ts, tw, key, windows, p.tlist[wi], sweep, jump, io, evals, partial, improved,
		                              max_shot);
	});
	if (lane == 0 && evals) {
		atomicAdd(counter, (unsigned long long)evals);
		if (partial) atomicAdd(counter + 1, (unsigned long long)partial);
	}
	if (metric_prop && lane == 0 && improved) atomicAdd(metric_prop, (unsigned long long)improved);
	if (metric_shots) {
		max_shot = __reduce_max_sync(kFull, max_shot);
		if (lane == 0 && max_shot >= 0) atomicMax(metric_shots, max_shot);
	}
}

// Jump distance of a sweep: 16, 8, 4, 2, 16, 8, ... (never above half the
// larger target side).
__host__ __device__ inline int jump_for(int sweep, int tW, int tH)
{
	int j = 16 >> (sweep % 4);
	while (j > 1 && 2 * j > max(tW, tH)) j /= 2;
	return j;
}

// Device buffers of the METRICS build's per-sweep figures (NULL: not kept).
struct PmMetrics {
	double *energy = nullptr;              // per sweep: sum of matched distances
	unsigned long long *prop = nullptr;    // per sweep: points improved by propagation
	int *shots = nullptr;                  // largest accepted draw index
	double *partials = nullptr;            // scratch of the energy reduction
	int partial_blocks = 0;
};

// Sum of the matched distances after a sweep (patchmatch.cu).
void sweep_energy(cudaStream_t s, const PmArgs &p, const float *dist, const PmMetrics &m, int sweep);

// The padded source as a tensor map of candidate windows (patchmatch.cu).
bool encode_source_map(const PmArgs &p, CUtensorMap *map);

template <int KIND, int C, int P, int NW>
__global__ void __launch_bounds__(32 * NW, team_blocks(NW))
    k_pm_sweep_team(DistArgs a, PmArgs p, int sweep, int jump, PmIo io, unsigned long long *counter,
                    unsigned long long *metric_prop, int *metric_shots)
{
	__shared__ PmTeam team;
	const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
	const PmSmem m = pm_smem<kPmGrouped>(a, p);
	unsigned *list = reinterpret_cast<unsigned *>(m.list);
	next_launch_may_start();
	load_weights(a, m.w);
	previous_launch_done();
	pm_count_clear(list);
	const uint2 key = pm_key(p);
	const int windows = 32 - __clz(p.max_window);
	int max_shot = -1;
	for (int i = blockIdx.x; i < p.nt; i += gridDim.x) {
		pm_sweep_team<KIND, C, P, NW>(p, m.w, list, &team, key, windows, p.tlist[i], sweep, jump, io, max_shot);
		__syncthreads();  // `team` is the next point's
	}
	pm_count_add(list, counter, nullptr);
	if (metric_prop && lane == 0 && pm_count(list)->improved)
		atomicAdd(metric_prop, (unsigned long long)pm_count(list)->improved);
	if (metric_shots && wid == 0) {
		max_shot = __reduce_max_sync(kFull, max_shot);
		if (lane == 0 && max_shot >= 0) atomicMax(metric_shots, max_shot);
	}
}

// The kernels' dynamic shared-memory limit is raised once per device, to the
// largest opt-in size (each launch passes the size it uses): a function
// attribute set on every call costs a driver call per PatchMatch call on
// every batch worker thread.
template <class Init, class Sweep>
static void raise_smem(nli_ctx *ctx, std::atomic<uint32_t> &raised, Init *init, Sweep *sweep)
{
	const uint32_t bit = 1u << (ctx->device & 31);
	if (raised.load(std::memory_order_acquire) & bit) return;
	NLI_CUDA(cudaFuncSetAttribute(init, cudaFuncAttributeMaxDynamicSharedMemorySize, ctx->max_smem_optin));
	NLI_CUDA(cudaFuncSetAttribute(sweep, cudaFuncAttributeMaxDynamicSharedMemorySize, ctx->max_smem_optin));
	raised.fetch_or(bit, std::memory_order_release);
}

// The one-point variants of the 9 x 9 kernels.
template <int KIND, int C, int P, int V>
static void launch_sweeps(nli_ctx *ctx, const DistArgs &a, const PmArgs &p, int iterations, const int2 *init,
                          const PmFields &b, unsigned long long *counter, const PmMetrics &mt,
                          const CUtensorMap &map, size_t smem)
{
	const PmShape shape = pm_shape(pm_threads(V), p.nt, ctx->num_sms);
	int *timeout = &ctx->status->timeout;
	static std::atomic<uint32_t> raised{0};  // one bit per device
	raise_smem(ctx, raised, k_pm_init<KIND, C, P, V>, k_pm_sweep<KIND, C, P, V>);
	NLI_REQUIRE(smem <= (size_t)ctx->max_smem_optin, NLI_E_UNSUPPORTED, "PatchMatch shared memory too large");
	{
		ProfScope ps(ctx, "pm_init");
		k_pm_init<KIND, C, P, V><<<shape.grid, shape.block, smem, ctx->stream>>>(a, p, init, b.nnf_x, b.dist_x,
		                                                                         counter, map, timeout);
		NLI_CHECK_LAUNCH();
	}
	for (int it = 0; it < iterations; it++) {
		ProfScope ps(ctx, "pm_sweep");
		k_pm_sweep<KIND, C, P, V><<<shape.grid, shape.block, smem, ctx->stream>>>(
		    a, p, it, jump_for(it, p.tW, p.tH), b.io(it), counter, mt.prop ? mt.prop + it : nullptr, mt.shots, map, timeout);
		NLI_CHECK_LAUNCH();
		if (mt.energy) sweep_energy(ctx->stream, p, b.io(it).dist_out, mt, it);
	}
}

template <int KIND, int C, int P>
static void launch_grouped(nli_ctx *ctx, const DistArgs &a, const PmArgs &p, int iterations, const int2 *init,
                           const PmFields &b, unsigned long long *counter, const PmMetrics &mt)
{
	const PmShape shape =
	    pm_shape(pm_threads(kPmGrouped), (p.nt + p.group.points - 1) / p.group.points, ctx->num_sms);
	const size_t smem = pm_smem_bytes(a.px * a.py, shape.block / 32);
	{
		ProfScope ps(ctx, "pm_init");
		launch_early(ctx->stream, shape.grid, shape.block, smem, k_pm_init_grouped<KIND, C, P>, a, p, init, b.nnf_x,
		             b.dist_x, counter);
		NLI_CHECK_LAUNCH();
	}
	const int team = pm_team(p.nt, ctx->num_sms);
	// Launched early a sweep loads its weights while the one before runs: about
	// 2 us less each, a call on 64 x 48 goes from 252 to 231 us, on 512 x 512
	// from 1378 to 1360, a run at 256 x 256 from 40.2 to 39.3 ms.  (The batch's
	// sweeps got slower this way, 8 images of 64 to 160 pixels 95 -> 109 ms, and
	// keep plain launches.)
	for (int it = 0; it < iterations; it++) {
		ProfScope ps(ctx, "pm_sweep");
		const int jump = jump_for(it, p.tW, p.tH);
		unsigned long long *prop = mt.prop ? mt.prop + it : nullptr;
		auto by_team = [&](auto nw) {
			constexpr int NW = decltype(nw)::value;
			const int grid = std::min(p.nt, team_blocks(NW) * ctx->num_sms);
			launch_early<true>(ctx->stream, grid, 32 * NW, pm_smem_bytes(a.px * a.py, NW),
			                   k_pm_sweep_team<KIND, C, P, NW>, a, p, it, jump, b.io(it), counter, prop, mt.shots);
		};
		if (team == 4)
			by_team(std::integral_constant<int, 4>());
		else if (team == 2)
			by_team(std::integral_constant<int, 2>());
		else
			launch_early<true>(ctx->stream, shape.grid, shape.block, smem, k_pm_sweep_grouped<KIND, C, P>, a, p, it,
			                   jump, b.io(it), counter, prop, mt.shots);
		NLI_CHECK_LAUNCH();
		if (mt.energy) sweep_energy(ctx->stream, p, b.io(it).dist_out, mt, it);
	}
}

// Fixed-size patches take the context's variant; the staged one only when
// the tensor map encodes and its layout fits, else (and for runtime-sized
// patches) kPmGrouped.
template <int KIND, int C, int P>
static void run_sweeps(nli_ctx *ctx, const DistArgs &a, PmArgs p, int iterations, const int2 *init,
                       const PmFields &b, unsigned long long *counter, const PmMetrics &mt)
{
	if constexpr (P == 9) {
		CUtensorMap map;
		std::memset(&map, 0, sizeof(map));
		const int taps = a.px * a.py, warps = pm_shape(pm_threads(ctx->tune_pm_variant), p.nt, ctx->num_sms).block / 32;
		if (ctx->tune_pm_variant == kPmStaged) {
			const size_t smem = pm_smem_bytes_tma(taps, p.rows, p.L, p.K, warps);
			if (smem <= (size_t)ctx->max_smem_optin && encode_source_map(p, &map)) {
				launch_sweeps<KIND, C, P, kPmStaged>(ctx, a, p, iterations, init, b, counter, mt, map, smem);
				return;
			}
		} else if (ctx->tune_pm_variant == kPmRegs) {
			launch_sweeps<KIND, C, P, kPmRegs>(ctx, a, p, iterations, init, b, counter, mt, map,
			                                   pm_smem_bytes(taps, warps));
			return;
		}
	}
	p.group = pm_group(p.nt, p.max_window, ctx->num_sms);
	launch_grouped<KIND, C, P>(ctx, a, p, iterations, init, b, counter, mt);
}

// ====================================================== batched launches
// PatchMatch calls of up to kBatchMax images in one launch per kernel (the
// lockstep batch driver, process.cu).  Every image is both source and
// target (as in the inpainting driver), with its own sizes, masks, target
// list, seed and call index; the distance, patch and PatchMatch parameters
// are shared.  Per target point the work is exactly that of the one-image
// kernels (the same device functions, Philox streams keyed by the image's
// own seed and call index), so each image's field equals its one-image
// call's bit for bit.
//
// The per-image arguments travel in the kernel's parameter space (a
// __grid_constant__ table read through the constant cache, not the L1 data
// pipe that bounds the sweep).  The persistent kernels see the concatenated
// target lists of the images still iterating (their `active` flag, written
// on the device between iterations) as one work list of groups (a group's
// points are one image's), distributed as the one-image kernels distribute
// theirs (pm_for_each: static block ranges or the device work queue).
struct PmBatchTask {
	PmArgs p;
	int flag;            // index of the image's active flag
	int moment_tiles;    // blocks of the image's bound tables
	unsigned long long *counter;  // the image's candidate counters (2)
	const float *img;    // the image (source = target), HWC float
	const int2 *init;    // initial field or null
	int2 *nnf_x;         // result
	PmIo io[2];          // even sweeps read x and write the second buffer, odd ones the other way round
};

struct PmBatchArgs {
	int n;
	const int *active;  // per image: still iterating (null: all)
	unsigned *queue;    // device work queue as PmArgs::queue (null: static ranges)
	int tile;
	PmGroup group;      // as PmArgs::group, the same for every image
	PmBatchTask t[kBatchMax];
};

__device__ __forceinline__ bool batch_on(const int *active, int t) { return !active || active[t] != 0; }

// Exclusive prefix of the active images' numbers of groups in s_pre[0..n]
// (s_pre[n] is the total); the whole block calls it.
__device__ __forceinline__ int pm_batch_prefix(const PmBatchArgs &B, int *s_pre)
{
	if (threadIdx.x < 32) {
		const int lane = threadIdx.x;
		const int t0 = 2 * lane, t1 = t0 + 1;
		auto groups = [&](int t) {
			return (t < B.n && batch_on(B.active, B.t[t].flag)) ? (B.t[t].p.nt + B.group.points - 1) / B.group.points
			                                                    : 0;
		};
		const int v0 = groups(t0), v1 = groups(t1);
		int incl = v0 + v1;
#pragma unroll
		for (int o = 1; o < 32; o <<= 1) {
			const int u = __shfl_up_sync(kFull, incl, o);
			if (lane >= o) incl += u;
		}
		const int excl = incl - v0 - v1;
		if (lane == 0) s_pre[0] = 0;
		s_pre[t0 + 1] = excl + v0;
		s_pre[t1 + 1] = excl + v0 + v1;
	}
	__syncthreads();
	return s_pre[B.n];
}

template <int KIND, int C, int P>
__global__ void __launch_bounds__(pm_threads(kPmGrouped), 1)
    k_pm_init_batch(DistArgs a, const __grid_constant__ PmBatchArgs B, unsigned long long *counter)
{
	__shared__ int s_pre[kBatchMax + 1];
	const PmSmem m = pm_smem<kPmGrouped>(a, B.t[0].p);
	load_weights(a, m.w);
	const int total = pm_batch_prefix(B, s_pre);
	const PmLane at = pm_lane(B.group);
	unsigned *list = reinterpret_cast<unsigned *>(m.list);
	pm_count_clear(list);
	int t = 0, tk = -1;
	uint2 key = make_uint2(0u, 0u);
	// a warp's items increase, so its image index only moves forward
	pm_for_each(total, B.queue, B.tile, [&](int i) {
		while (i >= s_pre[t + 1]) t++;
		const PmBatchTask &T = B.t[t];
		if (t != tk) {
			if (tk >= 0) {
				pm_count_add(list, counter, B.t[tk].counter);
				pm_count_clear(list);
			}
			key = pm_key(T.p);
			tk = t;
		}
		pm_init_group<KIND, C, P>(T.p, m.w, list, at, key, (i - s_pre[t]) * B.group.points, T.init, T.nnf_x,
		                          T.io[1].dist_out);
	});
	if (tk >= 0) pm_count_add(list, counter, B.t[tk].counter);
}

template <int KIND, int C, int P>
__global__ void __launch_bounds__(pm_threads(kPmGrouped), 1)
    k_pm_sweep_batch(DistArgs a, const __grid_constant__ PmBatchArgs B, int sweep, unsigned long long *counter)
{
	__shared__ int s_pre[kBatchMax + 1];
	const PmSmem m = pm_smem<kPmGrouped>(a, B.t[0].p);
	load_weights(a, m.w);
	const int total = pm_batch_prefix(B, s_pre);
	const PmLane at = pm_lane(B.group);
	unsigned *list = reinterpret_cast<unsigned *>(m.list);
	pm_count_clear(list);
	int max_shot = -1;
	int t = 0, tk = -1, windows = 0, jump = 1;
	uint2 key = make_uint2(0u, 0u);
	pm_for_each(total, B.queue ? B.queue + 1 + sweep : nullptr, B.tile, [&](int i) {
		while (i >= s_pre[t + 1]) t++;
		const PmBatchTask &T = B.t[t];
		if (t != tk) {
			if (tk >= 0) {
				pm_count_add(list, counter, B.t[tk].counter);
				pm_count_clear(list);
			}
			key = pm_key(T.p);
			windows = 32 - __clz(T.p.max_window);
			jump = jump_for(sweep, T.p.tW, T.p.tH);
			tk = t;
		}
		pm_sweep_group<KIND, C, P>(T.p, m.w, list, at, key, windows, (i - s_pre[t]) * B.group.points, sweep, jump,
		                           T.io[sweep & 1], max_shot);
	});
	if (tk >= 0) pm_count_add(list, counter, B.t[tk].counter);
}

template <int KIND, int C, int P>
static void run_batch_kernels(nli_ctx *ctx, const DistArgs &a, const PmBatchArgs &B, int iterations, long long groups,
                              unsigned long long *counter)
{
	const PmShape shape = pm_shape(pm_threads(kPmGrouped), groups, ctx->num_sms);
	const int block = shape.block, grid = shape.grid;
	const size_t smem = pm_smem_bytes(a.px * a.py, block / 32);
	{
		ProfScope ps(ctx, "pm_init");
		k_pm_init_batch<KIND, C, P><<<grid, block, smem, ctx->stream>>>(a, B, counter);
		NLI_CHECK_LAUNCH();
	}
	for (int it = 0; it < iterations; it++) {
		ProfScope ps(ctx, "pm_sweep");
		k_pm_sweep_batch<KIND, C, P><<<grid, block, smem, ctx->stream>>>(a, B, it, counter);
		NLI_CHECK_LAUNCH();
	}
}

// The kernels of one distance kind and channel count, compiled in a
// translation unit of their own (pm_*.cu).
template <int KIND, int C>
struct PmKernels {
	static void sweeps(nli_ctx *ctx, const DistArgs &a, const PmArgs &p, int iterations, const int2 *init,
	                   const PmFields &b, unsigned long long *counter, const PmMetrics &mt);
	static void batch(nli_ctx *ctx, const DistArgs &a, const PmBatchArgs &B, int iterations, long long groups,
	                  unsigned long long *counter);
};

#ifdef NLI_PM_INSTANTIATE
// Calls f with the patch side as a compile-time constant where the kernels
// are compiled for it (rows unrolled), else with 0.  Unrolling 7 x 7 took
// an L2-norm call on 425 x 283 from 614 to 522 us, 5 x 5 one on 285 x 518 from
// 448 to 399; other sizes keep the runtime loop.
template <class F>
void pm_sized(const DistArgs &a, F &&f)
{
	if (a.px == 9 && a.py == 9) return f(std::integral_constant<int, 9>());
	if (a.px == 7 && a.py == 7) return f(std::integral_constant<int, 7>());
	if (a.px == 5 && a.py == 5) return f(std::integral_constant<int, 5>());
	f(std::integral_constant<int, 0>());
}

template <int KIND, int C>
void PmKernels<KIND, C>::sweeps(nli_ctx *ctx, const DistArgs &a, const PmArgs &p, int iterations, const int2 *init,
                                const PmFields &b, unsigned long long *counter, const PmMetrics &mt)
{
	pm_sized(a, [&](auto size) { run_sweeps<KIND, C, decltype(size)::value>(ctx, a, p, iterations, init, b, counter, mt); });
}

template <int KIND, int C>
void PmKernels<KIND, C>::batch(nli_ctx *ctx, const DistArgs &a, const PmBatchArgs &B, int iterations, long long groups,
                               unsigned long long *counter)
{
	pm_sized(a, [&](auto size) {
		run_batch_kernels<KIND, C, decltype(size)::value>(ctx, a, B, iterations, groups, counter);
	});
}
#endif

// Calls f with the kernels of a distance kind and channel count; false when
// there are none.
template <class F>
bool pm_dispatch(int kind, int C, F &&f)
{
	if (kind == NLI_DIST_L2_RGBD && C == 4) return f(PmKernels<NLI_DIST_L2_RGBD, 4>()), true;
#define NLI_PM_CASE(KIND, CC) \
	if (kind == KIND && C == CC) return f(PmKernels<KIND, CC>()), true;
#define NLI_PM_CASES(KIND) NLI_PM_CASE(KIND, 1) NLI_PM_CASE(KIND, 2) NLI_PM_CASE(KIND, 3) NLI_PM_CASE(KIND, 4)
	NLI_PM_CASES(NLI_DIST_L2_COMBINED)
	NLI_PM_CASES(NLI_DIST_L2_NORM)
	NLI_PM_CASES(NLI_DIST_L1_NORM)
#undef NLI_PM_CASES
#undef NLI_PM_CASE
	return false;
}

// Records of the checked build's bounds tests, one per translation unit.
unsigned long long check_word_pm_combined();
unsigned long long check_word_pm_combined_rgb();
unsigned long long check_word_pm_rgbd();
unsigned long long check_word_pm_l2();
unsigned long long check_word_pm_l1();

}  // namespace nli
