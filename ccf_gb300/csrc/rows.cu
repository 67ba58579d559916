/******************************************************************************
rows.cu -- the full-sum Aberth solver with every row spread over the whole GPU:
the initial solve at the branch centres, and the full-sum continuation.

The sweep of solve_kernel (solver.cu, where the method is described), cut into
units of work that any CTA can take.  There a thread-block cluster owns a row:
a launch of few rows left most of the GPU idle (2 rows of 40 060 roots ran on
32 CTAs of 152 SMs, 67 ms), clusters of 8 share SMs unevenly, and each sweep
waits at the cluster's barrier for its slowest CTA (barrier the largest stall).
Here a row's sweep is two phases of independent units,

  step   64 to 256 roots of the row's list: the Aberth step from the sweep's
         correction sums, their snapshot, then the Newton check of the next
         sweep (f, f', and the roots whose Newton step is below the tolerance
         made final) and the unit's share of the next list;
  sums   one tile of targets against chunks of 1024 sources (roots, then
         stars): FP32 (FP64) partial sums per target, chunk and source share;

with a first check before them and the outputs (epilogue, and the next phi
step's first check) after them, both over blocks of 64 to 256 consecutive roots.  The
steps go over the list, not the row: after a few sweeps a block of the row
holds a handful of active roots and costs as much as a full one.  The list
keeps the row's order (each unit writes its survivors in order, and the CTA
that ends the phase joins the units' shares), so that neighbouring lanes hold
neighbouring roots: in the order of arrival the checks' leaf loops diverged
(the 20 000-star field's initial solve 14.8 ms against 12.8 over the row).  A CTA claims a unit from a row's ticket
(units and next unit in one 64-bit word); the CTA that finishes a
phase's last unit opens the next phase and keeps its first unit, and a phase
of one unit is not announced at all, so that a small row runs in one CTA
without a word in memory between its phases.  A CTA starts a row of its own while
rows are left, takes the units of that row, and helps other rows when its own
has none to give: rows of a batch run side by side, and one row alone spreads
over every SM.  No CTA waits for one that is not running: a phase's missing
units are held by CTAs at work, and a CTA without work may leave (it does
after POLL_LIMIT polls).

The results do not depend on the number of CTAs, nor on how the row is cut into
blocks and units: a unit's partial sums run over the same sources in the same
order, the chunks' FP32 sums are added in FP64 in chunk order, the source shares
S of a tile are those that solve_kernel's cluster of `cluster` CTAs would choose,
and every off-box point is summed by a 256-thread CTA (offbox_sums).  That is
the order of summation of solve_kernel, but for a block's off-box points beyond
OFF_CAP, which it leaves to a warp each.  (With another
order of summation a few rows in 1e5 trade roots: the iteration is chaotic
before it converges.)  The price is the partial sums in memory, 8 or 16 bytes
per target, chunk and share, so large launches run ROWS_PART_BYTES of rows at a
time, and a row of more than that alone has its units add their chunks up
(rows_plan.h); ccf_continue_branch_noalloc, which has no memory for them, keeps
solve_kernel.
******************************************************************************/
#define CCF_EVAL_UNROLL 4
#include "solver_dev.cuh"

#include <algorithm>
#include <atomic>

namespace ccf
{

namespace
{

enum RowPhase
{
	PHASE_FIRST = 0,   /* Newton check at a phi step's starting positions */
	PHASE_SUMS = 1,
	PHASE_STEP = 2,
	PHASE_EPILOGUE = 3
};

constexpr int POLL_LIMIT = 1 << 21;   /* polls in a row without work (~1 us each) after which a CTA leaves */

/* loads of what other CTAs wrote: past L1 */
CCF_D unsigned long long load_cg(const unsigned long long* p) { return __ldcg(p); }
CCF_D int load_volatile(const int* p) { return *(const volatile int*)p; }

/* shared memory of a CTA */
template <bool MIXED>
struct RowShared
{
	FieldView F;
	FieldOut O;
	RowDesc R;
	int row;                /* the row F, O, R belong to; -1: none */
	int cur;                /* the row this CTA started; -1: none */
	int unit, units, phase, it, j, total, late, split;
	int blk;                /* roots per unit of the phase (not of the sums) */
	SumsShape shape;
	int last;               /* this CTA finished the phase's last unit */
	int seg_blk;
	int seg_start[MAX_CLUSTER + 1];   /* of the row's segments, and their blocks of seg_blk before each */
	int seg_block[MAX_CLUSTER + 1];
	int phase_j;            /* the step that sphi, cphi belong to; -1: none */
	double sphi, cphi;
	int warp_list[NT / 32], warp_late[NT / 32];
	int own_next;           /* the next unit was kept by this CTA */
	int cand, claimed, started, quit;
	int noff, nan_err, nan_step;
	unsigned long long unconv;
	double maxerr;
	double2 offz[OFF_CAP];
	NearSums offs[OFF_CAP];
	__align__(16) typename Src<MIXED>::T buf[2 * CHUNK];
};
static_assert(OFF_CAP * (NT / 32) * 6 * sizeof(double) <= 2 * CHUNK * 16, "off-field scratch");

/* Star sums of the CTA's points off the root box (the threads with off set),
   each by the whole CTA, OFF_CAP of them at a time: which pass takes a point is
   no matter, its sum is the same wherever and with whatever others it is formed.
   Every thread calls it, with a barrier of the CTA between two calls. */
template <bool MIXED, bool NEED1, bool S3DF>
__device__ void offbox_sums(const FieldView& F, RowShared<MIXED>& S, bool off, double2 z, NearSums& sums)
{
	if (threadIdx.x == 0) S.noff = 0;
	__syncthreads();
	int q = -1;
	if (off)
	{
		q = atomicAdd(&S.noff, 1);
		if (q < OFF_CAP) S.offz[q] = z;
	}
	__syncthreads();
	const int n = S.noff;
	for (int q0 = 0; q0 < n; q0 += OFF_CAP)
	{
		const bool now = q >= q0 && q < q0 + OFF_CAP;
		if (q0 > 0)
		{
			if (now) S.offz[q - q0] = z;
			__syncthreads();
		}
		offfield_sums_cta<MIXED, NEED1, S3DF>(F, S.offz, min(n - q0, OFF_CAP), S.offs, reinterpret_cast<double*>(S.buf));
		if (now) sums = S.offs[q - q0];
	}
}

/* Newton check of a thread's root a at phase (cphi, sphi), at z: a root whose
   Newton step is under the tolerance takes it and is final; the others keep
   f and f' and go to the unit's share of the next list, in order; the final
   ones go to the share's end: their snapshot is due with the next step's (after
   the sums, as the others').  Every thread of the CTA calls it. */
template <bool MIXED>
__device__ void check_roots(const SolveArgs& A, RowShared<MIXED>& S, int* share, int* share_end, int* counts, int a, bool act, double2 z,
	double cphi, double sphi, bool initial)
{
	const FieldView& F = S.F;
	const long long base = S.R.base;
	const int leaf = act ? find_leaf(F, z) : 0;
	NearSums off = zero_sums();
	offbox_sums<MIXED, false, true>(F, S, act && leaf < 0, z, off);
	const FdF e = eval_fdf_warp<MIXED>(F, act, z, leaf, leaf < 0, off, cphi, sphi);
	bool still = act, late = false;
	if (act)
	{
		const double2 step = cdiv(e.f, e.df);
		if (isfinite(step.x) && isfinite(step.y) && hypot(step.x, step.y) < STEP_TOL * F.theta)
		{
			A.master[base + a] = csub(z, step);
			A.fin[base + a] = 1;
			still = false;
			late = true;
		}
		else
		{
			A.fval[2 * (base + a)] = e.f;
			A.fval[2 * (base + a) + 1] = e.df;
		}
	}
	const unsigned full = 0xffffffffu;
	const unsigned m = __ballot_sync(full, still), ml = __ballot_sync(full, late);
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
	if (lane == 0)
	{
		S.warp_list[warp] = __popc(m);
		S.warp_late[warp] = __popc(ml);
	}
	const int evals = __syncthreads_count(act);
	int g = __popc(m & ((1u << lane) - 1u)), gl = __popc(ml & ((1u << lane) - 1u)), n = 0, nl = 0;
	for (int w = 0; w < NT / 32; w++)
	{
		if (w < warp)
		{
			g += S.warp_list[w];
			gl += S.warp_late[w];
		}
		n += S.warp_list[w];
		nl += S.warp_late[w];
	}
	if (still) share[g] = a;
	if (late) share_end[-1 - gl] = a;
	if (threadIdx.x == 0)
	{
		if (counts)
		{
			*counts = n | nl << 16;
		}
		else
		{
			S.total = n;
			S.late = nl;
		}
		if (evals)
		{
			atomicAdd(&S.O.stats[2], (unsigned long long)evals);
			if (initial) atomicAdd(&S.O.stats[7], (unsigned long long)evals);
		}
	}
}

/* joins the units' shares into the row's list: the active roots in order from
   its start, the late ones from its end.  The whole CTA; the totals come back
   in Sh.total and Sh.late. */
template <bool MIXED>
__device__ void join_list(RowShared<MIXED>& S, const int* share, const int* counts, int units, int blk, int* list, int R)
{
	const unsigned full = 0xffffffffu;
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
	int carry = 0, carry_late = 0;
	for (int u0 = 0; u0 < units; u0 += NT)
	{
		const int u = u0 + threadIdx.x;
		const int v = u < units ? __ldcg(counts + u) : 0;
		const int n = v & 0xffff, nl = v >> 16;
		int x = n, y = nl;
		for (int o = 1; o < 32; o <<= 1)
		{
			const int xo = __shfl_up_sync(full, x, o), yo = __shfl_up_sync(full, y, o);
			if (lane >= o)
			{
				x += xo;
				y += yo;
			}
		}
		if (lane == 31)
		{
			S.warp_list[warp] = x;
			S.warp_late[warp] = y;
		}
		__syncthreads();
		int bx = carry, by = carry_late, tx = 0, ty = 0;
		for (int w = 0; w < NT / 32; w++)
		{
			if (w < warp)
			{
				bx += S.warp_list[w];
				by += S.warp_late[w];
			}
			tx += S.warp_list[w];
			ty += S.warp_late[w];
		}
		x += bx - n;    /* exclusive */
		y += by - nl;
		/* each warp copies its 32 units' shares, one unit at a time */
		const int most = min(32, units - u0 - warp * 32);
		for (int k = 0; k < most; k++)
		{
			const int kn = __shfl_sync(full, n, k), kl = __shfl_sync(full, nl, k);
			const int kx = __shfl_sync(full, x, k), ky = __shfl_sync(full, y, k);
			const int* from = share + (size_t)(u0 + warp * 32 + k) * blk;
			for (int i = lane; i < kn; i += 32) list[kx + i] = __ldcg(from + i);
			for (int i = lane; i < kl; i += 32) list[R - 1 - (ky + i)] = __ldcg(from + blk - 1 - i);
		}
		carry += tx;
		carry_late += ty;
		__syncthreads();
	}
	if (threadIdx.x == 0)
	{
		S.total = carry;
		S.late = carry_late;
	}
	__syncthreads();
}

/* the correction sums of an active root from the sweep's partial sums: the
   chunks of each source share in order, then the shares in order */
template <bool MIXED>
struct PartT
{
	using T = typename std::conditional<MIXED, float2, double2>::type;
};

/* float -> double (exact) on the integer pipe: the conversion instruction
   takes the FP64 pipe 64 cycles a warp, as many as the addition it feeds */
CCF_D double widen(float x)
{
	const unsigned u = __float_as_uint(x);
	const unsigned e = u & 0x7f800000u;
	if (e == 0u || e == 0x7f800000u) return (double)x;   /* zero, subnormal, infinite, NaN */
	return __hiloint2double((int)((u & 0x80000000u) | (((u & 0x7fffffffu) >> 3) + 0x38000000u)), (int)(u << 29));
}
CCF_D double widen(double x) { return x; }

/* one unit of the sums phase: tile against a group of chunks.  WHOLE: against
   all of them, the chunks of the roots and those of the stars added up in FP64
   in order, as gather_sums adds the chunks' sums. */
template <bool MIXED, int TP, bool WHOLE>
__device__ void sums_unit(const SolveArgs& A, RowShared<MIXED>& Sh, const int* list, typename PartT<MIXED>::T* part_out)
{
	using SrcT = typename Src<MIXED>::T;
	const FieldView& F = Sh.F;
	const int R = F.num_roots, N = F.num_stars;
	const long long base = Sh.R.base;
	const SrcT* rsrc;
	const SrcT* ssrc;
	if constexpr (MIXED)
	{
		rsrc = A.snap32 + base;
		ssrc = A.star_hilo[Sh.R.field];
	}
	else
	{
		rsrc = A.snap64 + base;
		ssrc = F.star_pos;
	}
	const int nrc = (R + CHUNK - 1) / CHUNK, nch = nrc + (N + CHUNK - 1) / CHUNK;
	const int S = Sh.split, total = Sh.total;
	const int tile = Sh.unit % Sh.shape.tiles, ch0 = Sh.unit / Sh.shape.tiles * Sh.shape.chunks;
	const int ch1 = min(ch0 + Sh.shape.chunks, nch);
	auto count = [&](int ch) { return ch < nrc ? min(CHUNK, R - ch * CHUNK) : min(CHUNK, N - (ch - nrc) * CHUNK); };
	auto issue = [&](int ch, int buf) {
		const SrcT* src = ch < nrc ? rsrc + (size_t)ch * CHUNK : ssrc + (size_t)(ch - nrc) * CHUNK;
		const int n = count(ch);
		for (int e = threadIdx.x; e < n; e += NT) cp_async16(&Sh.buf[buf * CHUNK + e], src + e);
		cp_async_commit();
	};
	issue(ch0, 0);
	const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
	const int part = warp % S, group = warp / S;
	const int groups = (Sh.shape.tpt == 0 ? HALF_WARPS : NT / 32) / S;   /* of 32 TP targets */
	/* a warp without a target only loads: it would take the others' issue slots */
	const bool work = group < groups && (tile * groups + group) * 32 * TP < total;
	int g[TP];
	SrcT zs[TP];
#pragma unroll
	for (int t = 0; t < TP; t++)
	{
		g[t] = work ? (tile * groups + group) * 32 * TP + t * 32 + lane : total;
		if constexpr (MIXED) zs[t] = g[t] < total ? __ldcg(rsrc + __ldcg(list + g[t])) : make_float4(0, 0, 0, 0);
		else zs[t] = g[t] < total ? __ldcg(rsrc + __ldcg(list + g[t])) : make_double2(0, 0);
	}
	double2 tot[WHOLE ? TP : 1];
	if constexpr (WHOLE)
	{
#pragma unroll
		for (int t = 0; t < TP; t++) tot[t] = make_double2(0, 0);
	}
	auto add_whole = [&](int t, int ch, double x, double y) {
		if constexpr (WHOLE)
		{
			tot[t].x += x;
			tot[t].y -= y;
			if (ch != nrc - 1 && ch != nch - 1) return;
			double2* whole = reinterpret_cast<double2*>(part_out) + (size_t)((ch < nrc ? 0 : S) + part) * total;
			if (g[t] < total) whole[g[t]] = tot[t];
			tot[t] = make_double2(0, 0);
		}
	};
	for (int ch = ch0; ch < ch1; ch++)
	{
		const int buf = (ch - ch0) & 1;
		if (ch + 1 < ch1) issue(ch + 1, buf ^ 1);
		else cp_async_commit();
		cp_async_wait<1>();
		__syncthreads();
		const int n = count(ch);
		const int j0 = (n * part) / S, j1 = work ? (n * (part + 1)) / S : j0;
		const SrcT* sb = Sh.buf + buf * CHUNK;
		typename PartT<MIXED>::T* out = part_out + ((size_t)ch * S + part) * total;
		if constexpr (MIXED)
		{
			float ax[TP], ay[TP];
#pragma unroll
			for (int t = 0; t < TP; t++) { ax[t] = 0.f; ay[t] = 0.f; }
#pragma unroll 4
			for (int jj = j0; jj < j1; jj++)
			{
				float4 s = sb[jj];
#pragma unroll
				for (int t = 0; t < TP; t++)
				{
					float dx = (zs[t].x - s.x) + (zs[t].z - s.z);
					float dy = (zs[t].y - s.y) + (zs[t].w - s.w);
					float d2 = fmaf(dx, dx, fmaf(dy, dy, 1e-30f));
					float r = rcp32(d2);
					ax[t] = fmaf(dx, r, ax[t]);
					ay[t] = fmaf(dy, r, ay[t]);
				}
			}
#pragma unroll
			for (int t = 0; t < TP; t++)
			{
				if constexpr (WHOLE) add_whole(t, ch, (double)ax[t], (double)ay[t]);
				else if (g[t] < total) out[g[t]] = make_float2(ax[t], ay[t]);
			}
		}
		else
		{
			double ax[TP], ay[TP];
#pragma unroll
			for (int t = 0; t < TP; t++) { ax[t] = 0; ay[t] = 0; }
#pragma unroll 2
			for (int jj = j0; jj < j1; jj++)
			{
				double2 s = sb[jj];
#pragma unroll
				for (int t = 0; t < TP; t++)
				{
					double dx = zs[t].x - s.x;
					double dy = zs[t].y - s.y;
					double d2 = fma(dx, dx, fma(dy, dy, 1e-300));
					double r = rcp64(d2);
					ax[t] = fma(dx, r, ax[t]);
					ay[t] = fma(dy, r, ay[t]);
				}
			}
#pragma unroll
			for (int t = 0; t < TP; t++)
			{
				if constexpr (WHOLE) add_whole(t, ch, ax[t], ay[t]);
				else if (g[t] < total) out[g[t]] = make_double2(ax[t], ay[t]);
			}
		}
		__syncthreads();
	}
}

/* out of line: only rows beyond ROWS_PART_BYTES take it */
template <bool MIXED>
__device__ __noinline__ void sums_unit_whole(const SolveArgs& A, RowShared<MIXED>& Sh, const int* list, typename PartT<MIXED>::T* part_out)
{
	if (Sh.shape.tpt <= 1) sums_unit<MIXED, 1, true>(A, Sh, list, part_out);
	else sums_unit<MIXED, TPT, true>(A, Sh, list, part_out);
}

/* The sums of position g of the row's list.  Every lane adds up its own root's,
   or, where the warp has few active roots and many chunks and shares, the
   lanes take one root together: lane 4 q + c the component c (roots x, y, stars
   x, y) of share q.  Either way a share's chunks are added in order, then the
   shares in order. */
template <bool MIXED>
CCF_D void gather_sums(const typename PartT<MIXED>::T* part, bool act, int g, int total, int S, int nrc, int nch, bool whole,
	double2& totR, double2& totS)
{
	const unsigned full = 0xffffffffu;
	totR = totS = make_double2(0, 0);
	if (whole)
	{
		/* the chunks are added up already (sums_unit) */
		if (!act) return;
		const double2* p = reinterpret_cast<const double2*>(part) + g;
		for (int q = 0; q < S; q++)
		{
			const double2 r = __ldcg(p + (size_t)q * total), s = __ldcg(p + (size_t)(S + q) * total);
			totR = q == 0 ? r : cadd(totR, r);
			totS = q == 0 ? s : cadd(totS, s);
		}
		return;
	}
	unsigned m = __ballot_sync(full, act);
	/* FP64 additions in a row: 2 per chunk and share; or the longer of the two
	   chunk ranges, the shares and the loads' latency (~10), per root */
	if (S * nch * 2 <= __popc(m) * (max(nrc, nch - nrc) + S + 10))
	{
		if (!act) return;
		for (int q = 0; q < S; q++)
		{
			double2 r = make_double2(0, 0), s = r;
			const typename PartT<MIXED>::T* p = part + (size_t)q * total + g;
			const size_t stride = (size_t)S * total;
#pragma unroll 4
			for (int ch = 0; ch < nrc; ch++)
			{
				const typename PartT<MIXED>::T v = __ldcg(p + ch * stride);
				r.x += widen(v.x);
				r.y -= widen(v.y);
			}
#pragma unroll 4
			for (int ch = nrc; ch < nch; ch++)
			{
				const typename PartT<MIXED>::T v = __ldcg(p + ch * stride);
				s.x += widen(v.x);
				s.y -= widen(v.y);
			}
			totR = q == 0 ? r : cadd(totR, r);
			totS = q == 0 ? s : cadd(totS, s);
		}
		return;
	}
	const int lane = threadIdx.x & 31;
	const int q = min(lane >> 2, S - 1), c = lane & 3;
	const int c0 = c < 2 ? 0 : nrc, c1 = c < 2 ? nrc : nch;
	while (m)
	{
		const int src = __ffs(m) - 1;
		m &= m - 1;
		const int gg = __shfl_sync(full, g, src);
		double t = 0;
#pragma unroll 4
		for (int ch = c0; ch < c1; ch++)
		{
			const typename PartT<MIXED>::T p = __ldcg(part + ((size_t)ch * S + q) * total + gg);
			if (c & 1) t -= widen(p.y);
			else t += widen(p.x);
		}
		/* lanes 0 .. 3 add their component's shares */
		double v = t;
		for (int s = 1; s < S; s++) v += __shfl_sync(full, t, 4 * s + c);
		const double rx = __shfl_sync(full, v, 0), ry = __shfl_sync(full, v, 1);
		const double sx = __shfl_sync(full, v, 2), sy = __shfl_sync(full, v, 3);
		if (lane == src)
		{
			totR = make_double2(rx, ry);
			totS = make_double2(sx, sy);
		}
	}
}

template <bool MIXED>
__global__ void __launch_bounds__(NT, 2) rows_kernel(const SolveArgs A, const int initial)
{
	__shared__ RowShared<MIXED> Sh;
	const int num_rows = A.num_rows_dev ? min(*A.num_rows_dev, A.num_rows) : A.num_rows;
	if (num_rows == 0) return;
	const int csize = A.cluster;
	const int rows_at_work = min(num_rows, A.part_slots);
	if (threadIdx.x == 0)
	{
		Sh.row = -1;
		Sh.cur = -1;
		Sh.own_next = 0;
	}
	int polls = 0;
	__syncthreads();

	while (true)
	{
		/* the kept unit; else claim one: of this CTA's own row, of a row it starts,
		   else of any row.  A ticket is read before it is drawn from, so that
		   polling does not count it up. */
		auto claim = [&](int r) {
			RowState* st = A.state + r;
			const unsigned long long t = load_cg(&st->ticket);
			if (ticket_next(t) >= ticket_units(t)) return false;
			const unsigned long long u = atomicAdd(&st->ticket, 1ull);
			if (ticket_next(u) >= ticket_units(u)) return false;
			__threadfence();
			Sh.unit = ticket_next(u);
			Sh.units = ticket_units(u);
			Sh.claimed = r;
			Sh.phase = load_volatile(&st->phase);
			Sh.it = load_volatile(&st->it);
			Sh.j = load_volatile(&st->j);
			Sh.total = load_volatile(&st->total);
			Sh.late = load_volatile(&st->late);
			Sh.split = load_volatile(&st->split);
			Sh.blk = load_volatile(&st->blk);
			Sh.shape.tpt = load_volatile(&st->tpt);
			Sh.shape.chunks = load_volatile(&st->chunks);
			Sh.shape.tiles = load_volatile(&st->tiles);
			Sh.shape.whole = load_volatile(&st->whole);
			return true;
		};
		const bool kept = Sh.own_next != 0;
		__syncthreads();
		if (!kept)
		{
			if (threadIdx.x == 0)
			{
				Sh.unit = -1;
				Sh.cand = 1 << 30;
				Sh.quit = 0;
				if (Sh.cur >= 0 && load_volatile(&A.state[Sh.cur].complete)) Sh.cur = -1;
				bool got = Sh.cur >= 0 && claim(Sh.cur);
				if (!got && Sh.cur < 0)
				{
					const int nr = load_volatile(&A.control[0]);
					/* a row waits for its slot of the partial sums */
					if (nr < num_rows && (nr < A.part_slots || load_volatile(&A.state[nr - A.part_slots].complete)) &&
						atomicCAS(&A.control[0], nr, nr + 1) == nr)
					{
						__threadfence();
						const RowDesc rd = A.rows[nr];
						RowState* st = A.state + nr;
						const int first = initial ? 0 : A.outs[rd.field].step_first, last = initial ? 0 : rd.steps;
						if (first > last)
						{
							/* no steps to run */
							atomicAdd(&A.outs[rd.field].stats[STAT_ROWS_DONE], 1ull);
							st->complete = 1;
							__threadfence();
							atomicAdd(&A.control[1], 1);
						}
						else
						{
							const int nr0 = A.fields[rd.field].num_roots, blk = block_roots(nr0, rows_at_work, (int)gridDim.x, A.fields[rd.field].rectangular != 0);
							const int units = row_blocks(nr0, csize, blk);
							Sh.cur = nr;
							Sh.claimed = nr;
							Sh.unit = 0;
							Sh.units = units;
							Sh.phase = PHASE_FIRST;
							Sh.it = 0;
							Sh.j = first;
							Sh.total = Sh.late = 0;
							Sh.split = 1;
							Sh.blk = blk;
							got = true;
							/* the state is zero: phase, it, counts */
							st->j = first;
							st->blk = blk;
							if (units > 1)
							{
								__threadfence();
								atomicExch(&st->ticket, ticket_open(units) | 1ull);
							}
						}
					}
				}
				if (!got && load_volatile(&A.control[1]) >= num_rows) Sh.quit = 1;
				Sh.started = min(load_volatile(&A.control[0]), num_rows);
			}
			__syncthreads();
			if (Sh.quit) break;
			if (Sh.unit < 0)
			{
				/* the nearest started row with a unit left, from this CTA's place on */
				const int started = Sh.started;
				for (int k = threadIdx.x; k < started; k += NT)
				{
					const unsigned long long t = load_cg(&A.state[(blockIdx.x + (unsigned)k) % (unsigned)started].ticket);
					if (ticket_next(t) < ticket_units(t))
					{
						atomicMin(&Sh.cand, k);
						break;
					}
				}
				__syncthreads();
				if (threadIdx.x == 0 && Sh.cand < (1 << 30)) claim((int)((blockIdx.x + (unsigned)Sh.cand) % (unsigned)started));
				__syncthreads();
				if (Sh.unit < 0)
				{
					if (++polls > POLL_LIMIT) break;
					__nanosleep(200);
					__syncthreads();
					continue;
				}
			}
		}
		polls = 0;
		const int row = Sh.claimed;
		RowState* st = A.state + row;
		if (Sh.row != row)
		{
			__syncthreads();   /* everyone has compared Sh.row */
			const RowDesc* rd = A.rows + row;
			const int field = rd->field;
			auto copy = [&](void* dst, const void* src, int bytes) {
				for (int i = threadIdx.x; i < bytes / 4; i += NT) ((int*)dst)[i] = ((const int*)src)[i];
			};
			static_assert(sizeof(FieldView) % 4 == 0 && sizeof(FieldOut) % 4 == 0 && sizeof(RowDesc) % 4 == 0, "word copies");
			copy(&Sh.F, A.fields + field, sizeof(FieldView));
			copy(&Sh.O, A.outs + field, sizeof(FieldOut));
			copy(&Sh.R, rd, sizeof(RowDesc));
			if (threadIdx.x <= csize) Sh.seg_start[threadIdx.x] = segment_start(A.fields[field].num_roots, csize, threadIdx.x);
			if (threadIdx.x == 0)
			{
				Sh.row = row;
				Sh.phase_j = -1;
			}
			__syncthreads();
			if (threadIdx.x == 0)
			{
				const int blk = block_roots(A.fields[field].num_roots, rows_at_work, (int)gridDim.x, A.fields[field].rectangular != 0);
				int n = 0;
				for (int r = 0; r < csize; r++)
				{
					Sh.seg_block[r] = n;
					n += (Sh.seg_start[r + 1] - Sh.seg_start[r] + blk - 1) / blk;
				}
				Sh.seg_block[csize] = n;
				Sh.seg_blk = blk;
			}
		}
		const FieldView& F = Sh.F;
		const FieldOut& O = Sh.O;
		const int R = F.num_roots, N = F.num_stars;
		const long long base = Sh.R.base;
		const int c = Sh.R.branch, side = Sh.R.side;
		const int nrc = (R + CHUNK - 1) / CHUNK, nch = nrc + (N + CHUNK - 1) / CHUNK;
		const int max_it = initial ? O.max_iters_init : O.max_iters_step;
		const int j1 = initial ? 0 : Sh.R.steps;
		if (threadIdx.x == 0)
		{
			Sh.own_next = 0;
			Sh.nan_err = 0;
			Sh.nan_step = 0;
			Sh.unconv = 0;
			Sh.maxerr = 0;
			if (Sh.phase != PHASE_SUMS && Sh.phase_j != Sh.j)
			{
				const double phi = initial ? (PI / O.nb + c * 2 * PI / O.nb) : row_phi(c, O.nb, O.nphi, side, Sh.j);
				sincos(phi, &Sh.sphi, &Sh.cphi);
				Sh.phase_j = Sh.j;
			}
		}
		__syncthreads();
		int* const list = A.list + base;
		int* const shares = A.share + (size_t)(row % A.part_slots) * A.share_stride;
		int* const counts = A.counts + (size_t)(row % A.part_slots) * A.counts_stride;
		const int blk = Sh.blk, tid = threadIdx.x < blk ? (int)threadIdx.x : NO_ROOT;
		/* the unit's share of the next list; the list itself when it is the only unit */
		const bool only = Sh.units == 1;
		int* const share = only ? list : shares + (size_t)Sh.unit * blk;
		int* const share_end = only ? list + R : share + blk;
		int* const share_count = only ? nullptr : counts + Sh.unit;
		typename PartT<MIXED>::T* part = reinterpret_cast<typename PartT<MIXED>::T*>(
			reinterpret_cast<unsigned char*>(A.part) + (size_t)(row % A.part_slots) * A.part_stride);

		if (Sh.phase == PHASE_SUMS)
		{
			if (Sh.shape.whole) sums_unit_whole<MIXED>(A, Sh, list, part);
			else if (Sh.shape.tpt <= 1) sums_unit<MIXED, 1, false>(A, Sh, list, part);
			else sums_unit<MIXED, TPT, false>(A, Sh, list, part);
		}
		else
		{
			const int j = Sh.j;
			double sphi = Sh.sphi, cphi = Sh.cphi;
			if (Sh.phase == PHASE_STEP)
			{
				/* the roots of the list, then those made final by the last check */
				const int g = Sh.unit * blk + threadIdx.x, total = Sh.total;
				const bool own = tid < NO_ROOT && g < total + Sh.late;
				bool act = own && g < total;
				const int a = own ? __ldcg(list + (act ? g : R - 1 - (g - total))) : 0;
				double2 z = own ? __ldcg(A.master + base + a) : make_double2(0, 0);
				double2 totR, totS;
				gather_sums<MIXED>(part, act, g, total, Sh.split, nrc, nch, Sh.shape.whole != 0, totR, totS);
				if (act)
				{
					const double2 f = __ldcg(A.fval + 2 * (base + a)), df = __ldcg(A.fval + 2 * (base + a) + 1);
					double2 Sg = make_double2(2 * totS.x - totR.x, 2 * totS.y - totR.y);
					if (!F.rectangular && !F.approx)
					{
						const double2 iz = cinv(z);
						Sg.x += 2 * iz.x;
						Sg.y += 2 * iz.y;
					}
					const double2 znew = csub(z, cdiv(f, cadd(df, cmul(f, Sg))));
					if (isfinite(znew.x) && isfinite(znew.y))
					{
						A.master[base + a] = znew;
						if (hypot(znew.x - z.x, znew.y - z.y) < STEP_TOL * F.theta)
						{
							A.fin[base + a] = 1;
							act = false;
						}
						z = znew;
					}
					else
					{
						A.fin[base + a] = 2;   /* frozen: counted as unconverged */
						Sh.nan_step = 1;
						act = false;
					}
				}
				if (own)
				{
					if constexpr (MIXED) A.snap32[base + a] = split_hilo(z);
					else A.snap64[base + a] = z;
				}
				if (Sh.it < max_it) check_roots<MIXED>(A, Sh, share, share_end, share_count, a, act, z, cphi, sphi, initial);
			}
			else
			{
				/* the block's roots */
				int r = 0;
				while (r + 1 < csize && Sh.unit >= Sh.seg_block[r + 1]) r++;
				const int a = Sh.seg_start[r] + (Sh.unit - Sh.seg_block[r]) * blk + threadIdx.x;
				const int o1 = Sh.seg_start[r + 1];
				const bool own = tid < NO_ROOT && a < o1;
				const double2 z = own ? __ldcg(A.master + base + a) : make_double2(0, 0);
				bool check = true;
				if (Sh.phase == PHASE_EPILOGUE)
				{
					/* outputs of this phi step */
					int ob[2] = {c, c}, ok[2] = {O.half, 0};
					const int nslot = initial ? 1 : row_slots(O.nb, O.half, O.seg, c, side, j, ob, ok);
					const int leaf = own ? find_leaf(F, z) : 0;
					NearSums off = zero_sums();
					if (O.mu) offbox_sums<MIXED, true, true>(F, Sh, own && leaf < 0, z, off);
					else offbox_sums<MIXED, true, false>(F, Sh, own && leaf < 0, z, off);
					const size_t out = out_slot(O, own ? a : 0, ob[0], ok[0]);
					const size_t out2 = nslot > 1 ? out_slot(O, own ? a : 0, ob[1], ok[1]) : NO_SLOT;
					const bool unconv = own && __ldcg(A.fin + base + a) != 1;
					if (!point_epilogue_warp<MIXED>(F, O, own, z, leaf, leaf < 0, off, out, out2, cphi, sphi, &Sh.maxerr, unconv))
						Sh.nan_err = 1;
					if (unconv) atomicAdd(&Sh.unconv, 1ull);
					if (own && initial)
					{
						const long long cb = Sh.R.cont_base;
						O.cont_master[cb + a] = z;
						O.cont_master[cb + R + a] = z;
						if constexpr (MIXED)
						{
							const float4 h = split_hilo(z);
							O.cont_snap32[cb + a] = h;
							O.cont_snap32[cb + R + a] = h;
						}
						else
						{
							O.cont_snap64[cb + a] = z;
							O.cont_snap64[cb + R + a] = z;
						}
					}
					check = j < j1;
					if (check)
					{
						/* the next step's first check */
						__syncthreads();
						if (threadIdx.x == 0)
						{
							sincos(row_phi(c, O.nb, O.nphi, side, j + 1), &Sh.sphi, &Sh.cphi);
							Sh.phase_j = j + 1;
						}
						__syncthreads();
						sphi = Sh.sphi;
						cphi = Sh.cphi;
					}
				}
				if (check)
				{
					if (own) A.fin[base + a] = 0;
					check_roots<MIXED>(A, Sh, share, share_end, share_count, a, own, z, cphi, sphi, initial);
				}
			}
		}

		/* the unit is done: its writes, then the count; the phase's last unit opens
		   the next phase.  (checked: the phase made a list; read before thread 0
		   moves on.) */
		const bool checked = (Sh.phase == PHASE_STEP && Sh.it < max_it) || Sh.phase == PHASE_FIRST ||
			(Sh.phase == PHASE_EPILOGUE && Sh.j < j1);
		__syncthreads();
		if (threadIdx.x == 0)
		{
			unsigned long long* stats = O.stats;
			if (Sh.maxerr > 0) atomicMax(&stats[0], (unsigned long long)__double_as_longlong(Sh.maxerr));
			const unsigned long long flags = (Sh.nan_err ? 1ull : 0ull) | (Sh.nan_step ? 2ull : 0ull);
			if (flags) atomicOr(&stats[1], flags);
			if (Sh.unconv) atomicAdd(&stats[4], Sh.unconv);
			int last = Sh.units == 1;
			if (!last)
			{
				__threadfence();
				last = atomicAdd(&st->done, 1) == Sh.units - 1;
				if (last)
				{
					__threadfence();
					st->done = 0;
				}
			}
			Sh.last = last;
		}
		__syncthreads();
		if (!Sh.last) continue;
		/* the next phase (only, like checked, was read before: without a list to
		   join thread 0 moves on at once) */
		if (checked && !only) join_list<MIXED>(Sh, shares, counts, Sh.units, blk, list, R);
		if (threadIdx.x == 0)
		{
			unsigned long long* stats = O.stats;
			int phase = Sh.phase, units = 0;
			if (phase == PHASE_SUMS)
			{
				phase = PHASE_STEP;
				Sh.it++;
				Sh.blk = block_roots(Sh.total + Sh.late, rows_at_work, (int)gridDim.x, F.rectangular != 0);
				units = (Sh.total + Sh.late + Sh.blk - 1) / Sh.blk;
			}
			else
			{
				if (phase == PHASE_EPILOGUE)
				{
					atomicMax(&stats[initial ? 5 : 6], (unsigned long long)Sh.it);
					Sh.j++;
					Sh.it = 0;
				}
				if (Sh.j > j1)
				{
					atomicAdd(&stats[STAT_ROWS_DONE], 1ull);
					__threadfence();
					st->complete = 1;
					__threadfence();
					atomicAdd(&A.control[1], 1);
				}
				else if (checked && Sh.total > 0)
				{
					phase = PHASE_SUMS;
					Sh.split = source_split(Sh.total, csize);
					Sh.shape = sums_shape(Sh.total, Sh.split, R, N, nch, rows_at_work, (int)gridDim.x / 2,
						sums_whole(Sh.total, Sh.split, nch, MIXED, A.part_limit));
					units = Sh.shape.tiles * Sh.shape.groups;
					const unsigned long long terms = (unsigned long long)Sh.total * (unsigned long long)(R - 1 + N);
					atomicAdd(&stats[3], terms);
					if (initial) atomicAdd(&stats[8], terms);
				}
				else
				{
					phase = PHASE_EPILOGUE;
					Sh.blk = Sh.seg_blk;
					units = Sh.seg_block[csize];
				}
			}
			if (units > 0)
			{
				Sh.phase = phase;
				Sh.unit = 0;
				Sh.units = units;
				Sh.own_next = 1;
				if (units > 1)
				{
					st->phase = phase;
					st->it = Sh.it;
					st->j = Sh.j;
					st->total = Sh.total;
					st->late = Sh.late;
					st->split = Sh.split;
					st->blk = Sh.blk;
					st->tpt = Sh.shape.tpt;
					st->chunks = Sh.shape.chunks;
					st->tiles = Sh.shape.tiles;
					st->whole = Sh.shape.whole;
					__threadfence();
					atomicExch(&st->ticket, ticket_open(units) | 1ull);
				}
			}
		}
		__syncthreads();
	}
}

}

cudaError_t launch_rows(cudaStream_t s, const SolveArgs& a, bool mixed, bool initial, int num_sms, int max_roots, int max_stars)
{
	if (a.num_rows == 0) return cudaSuccess;
	static std::atomic<int> known[2];
	int per_sm = known[mixed ? 1 : 0].load(std::memory_order_relaxed);
	if (per_sm == 0)
	{
		if (mixed) cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, rows_kernel<true>, NT, 0);
		else cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, rows_kernel<false>, NT, 0);
		per_sm = std::max(per_sm, 1);
		known[mixed ? 1 : 0].store(per_sm, std::memory_order_relaxed);
	}
	/* as many CTAs as the rows can ever have units for */
	const long long chunks = (max_roots + CHUNK - 1) / CHUNK + (max_stars + CHUNK - 1) / CHUNK;
	const long long units = std::max<long long>(max_roots / MIN_BLOCK + a.cluster, chunks * ((max_roots + 31) / 32));
	const int blocks = (int)std::min<long long>((long long)num_sms * per_sm, units * a.num_rows);
	if (mixed) rows_kernel<true><<<blocks, NT, 0, s>>>(a, initial ? 1 : 0);
	else rows_kernel<false><<<blocks, NT, 0, s>>>(a, initial ? 1 : 0);
	return cudaGetLastError();
}

} /* namespace ccf */
