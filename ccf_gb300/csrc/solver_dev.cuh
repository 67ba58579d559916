/******************************************************************************
solver_dev.cuh -- device functions shared by the full-sum solvers (solver.cu,
rows.cu) and the tracker: the evaluation of f and f' of a warp's roots, the
outputs of a final root, and the CTA-wide star sums of points off the root
box.
******************************************************************************/
#pragma once

#include "field_df.cuh"
#include "kernels.h"
#include "rows_plan.h"

#include <type_traits>

namespace ccf
{

CCF_D void cp_async16(void* smem, const void* gmem)
{
	unsigned s = (unsigned)__cvta_generic_to_shared(smem);
	asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(s), "l"(gmem) : "memory");
}
CCF_D void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
CCF_D void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

template <bool MIXED>
struct Src
{
	using T = typename std::conditional<MIXED, float4, double2>::type;
};

constexpr int OFF_CAP = 64;      /* off-field points summed by the CTA per pass */

/* Star sums of the off-field points pts[0..K), K <= OFF_CAP.  A point outside
   the root box takes the direct sum over every star, as in the reference
   (include/tree_node.cuh:535-539, include/alpha_star.cuh:26-37).  The whole
   CTA works on each point: every thread takes every NT-th star, the warps
   reduce by shuffles and the per-warp partials meet in shared memory (red,
   K * NT/32 * 6 doubles).  MIXED evaluates in double-float on the FP32 pipe
   from the split star arrays, s3 in double-float only when S3DF; otherwise
   FP64.  All threads of the CTA must call it; it ends with a barrier, after
   which out[0..K) holds the sums. */
template <bool MIXED, bool NEED1, bool S3DF>
__device__ void offfield_sums_cta(const FieldView& F, const double2* pts, int K, NearSums* out, double* red)
{
	const unsigned full = 0xffffffffu;
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
	for (int k = 0; k < K; k++)
	{
		double v[6];
		if constexpr (MIXED)
		{
			const dfc z = dfc_from(pts[k]);
			SumsDF a;
			a.s1 = {{0.f, 0.f}, {0.f, 0.f}};
			a.s2 = a.s1;
			dfc s3 = a.s1;
			float2 s3f = make_float2(0.f, 0.f);
			for (int i = threadIdx.x; i < F.num_stars; i += NT)
				star_term_df<NEED1, S3DF>(a, s3, s3f, z, F.star_df[i], F.star_mass_df[i]);
			if (!S3DF) s3 = {{s3f.x, 0.f}, {s3f.y, 0.f}};
			dfl w[6] = {a.s1.re, a.s1.im, a.s2.re, a.s2.im, s3.re, s3.im};
#pragma unroll
			for (int c = 0; c < 6; c++)
			{
				for (int o = 16; o > 0; o >>= 1)
				{
					dfl u = {__shfl_xor_sync(full, w[c].hi, o), __shfl_xor_sync(full, w[c].lo, o)};
					w[c] = df_add(w[c], u);
				}
				v[c] = df_to_double(w[c]);
			}
		}
		else
		{
			NearSums a = zero_sums();
			for (int i = threadIdx.x; i < F.num_stars; i += NT)
			{
				const double2 p = F.star_pos[i];
				star_term<NEED1, true>(a, pts[k], p.x, p.y, F.star_mass[i]);
			}
			double u[6] = {a.s1.x, a.s1.y, a.s2.x, a.s2.y, a.s3.x, a.s3.y};
#pragma unroll
			for (int c = 0; c < 6; c++)
			{
				for (int o = 16; o > 0; o >>= 1) u[c] += __shfl_xor_sync(full, u[c], o);
				v[c] = u[c];
			}
		}
		if (lane == 0)
		{
#pragma unroll
			for (int c = 0; c < 6; c++) red[(k * (NT / 32) + warp) * 6 + c] = v[c];
		}
	}
	__syncthreads();
	if (threadIdx.x < K)
	{
		const int k = threadIdx.x;
		double v[6] = {0, 0, 0, 0, 0, 0};
		for (int q = 0; q < NT / 32; q++)
		{
#pragma unroll
			for (int c = 0; c < 6; c++) v[c] += red[(k * (NT / 32) + q) * 6 + c];
		}
		out[k].s1 = make_double2(v[0], v[1]);
		out[k].s2 = make_double2(v[2], v[3]);
		out[k].s3 = make_double2(v[4], v[5]);
	}
	__syncthreads();
}

/* phase of step j of a row (include/ccf_functions.cuh:338-344) */
CCF_D double row_phi(int c, int nb, int nphi, int side, int j)
{
	double phi0 = PI / nb + c * 2 * PI / nb;
	double dphi = 2 * PI / nphi * j;
	return side == 0 ? phi0 - dphi : phi0 + dphi;
}

/* f and f' of a root */
struct FdF
{
	double2 f, df;
};

/* f(z; phi) and f'(z) for the root of every lane with valid set, given its
   leaf.  An off-field root (leaf < 0) takes its star sums from off when
   have_off is set (the CTA computed them) and otherwise from the whole warp
   -- so all 32 lanes of the warp must call it.  Not inlined: the evaluation
   needs its registers once, not in every caller's frame. */
template <bool MIXED>
static __device__ __noinline__ FdF eval_fdf_warp(const FieldView& F, bool valid, double2 z, int leaf, bool have_off, NearSums off,
	double cphi, double sphi)
{
	NearSums ns = have_off ? off : zero_sums();
	if (!MIXED && valid && leaf >= 0) ns = leaf_sums<false, true>(F, leaf, z);
	offfield_sums_warp<false, true>(F, valid && leaf < 0 && !have_off, z, ns);
	FdF r;
	r.f = make_double2(0, 0);
	r.df = make_double2(0, 0);
	if (!valid) return r;
	if constexpr (MIXED)
	{
		/* f in double-float on the FP32 pipe, off-field points included;
		   f' in FP32, or FP64 where FP32 overflows */
		eval_fdf_df(F, leaf, z, cphi, sphi, ns, r.f, r.df);
	}
	else
	{
		eval_f64<true>(F, leaf, z, cphi, sphi, ns, r.f, r.df);
	}
	return r;
}

/* A root is final once its step is below this many theta_star (the
   reference's test, include/ccf_functions.cuh:385). */
constexpr double STEP_TOL = 0.000000001;

/* outputs of one final root per lane: position, 1/mu bound, caustic,
   length scale; returns false when the 1/mu bound is not finite.  All 32
   lanes must call it (see aberth_update_warp for leaf, have_off and off).
   With DF and no length scales every point is evaluated in double-float (off
   the root box from the star sums); length scales use FP64. */
constexpr size_t NO_SLOT = ~(size_t)0;

template <bool DF>
static __device__ __noinline__ bool point_epilogue_warp(const FieldView& F, const FieldOut& O, bool valid, double2 z, int leaf,
	bool have_off, NearSums off, size_t out, size_t out2, double cphi, double sphi, double* maxerr, bool unconv)
{
	NearSums ns = have_off ? off : zero_sums();
	const bool mu = O.mu != nullptr;
	const bool use_df = DF && !mu;
	if (!use_df && valid && leaf >= 0) ns = mu ? leaf_sums<true, true>(F, leaf, z) : leaf_sums<true, false>(F, leaf, z);
	offfield_sums_warp<true, true>(F, valid && leaf < 0 && !have_off, z, ns);
	if (!valid) return true;
	PointResult pr;
	if (use_df) pr = eval_point_df(F, leaf, z, cphi, sphi, ns);
	else if (O.caustics && mu) pr = eval_point<true, true>(F, leaf, z, cphi, sphi, ns);
	else if (O.caustics) pr = eval_point<true, false>(F, leaf, z, cphi, sphi, ns);
	else if (mu) pr = eval_point<false, true>(F, leaf, z, cphi, sphi, ns);
	else pr = eval_point<false, false>(F, leaf, z, cphi, sphi, ns);
	/* an unconverged point is marked for the FP64 polish (polish.cu) */
	const double stored = unconv ? unconverged_mark(pr.err) : pr.err;
	if (out != NO_SLOT)
	{
		O.ccs[out] = z;
		O.errs[out] = stored;
		if (O.caustics) O.caustics[out] = pr.w;
		if (mu) O.mu[out] = pr.mu_length;
	}
	if (out2 != NO_SLOT)
	{
		O.ccs[out2] = z;
		O.errs[out2] = stored;
		if (O.caustics) O.caustics[out2] = pr.w;
		if (mu) O.mu[out2] = pr.mu_length;
	}
	if (!isfinite(pr.err)) return false;
	atomicMax((unsigned long long*)maxerr, (unsigned long long)__double_as_longlong(pr.err));
	return true;
}

} /* namespace ccf */
