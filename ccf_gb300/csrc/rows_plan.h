/******************************************************************************
rows_plan.h -- how the full-sum solver's work is cut: the CTA's shape, the
blocks and units of a row (rows.cu), and the ticket its units are drawn from.
Host and device code, so that the plan can be checked on the host.
******************************************************************************/
#pragma once

#include "common.cuh"

#include <algorithm>

namespace ccf
{

constexpr int NT = 256;          /* threads per CTA */
constexpr int MAX_SOLVE_CLUSTER = 8;   /* CTAs per row of solve_kernel (the portable cluster sizes) */
constexpr int MAX_CLUSTER = 16;  /* and of the clusters whose order of summation rows_kernel keeps */
constexpr int TPT = 2;           /* targets per thread */
constexpr int TILE = NT * TPT;   /* targets per tile */
constexpr int CHUNK = 1024;      /* sources per shared-memory stage */

constexpr int CLUSTER_CTAS_PER_SM = 2;   /* CTAs of such a cluster that an SM holds (the rule of the order
                                            of summation, Engine::solve, fills the GPU with them once) */

/* ticket of a row: the units of the open phase and the next unit (0: none) in
   one word, each as wide as the int it is read into (of 22 bits a first sweep
   of 610 000 stars, 4.3e6 units, left 66 000) */
constexpr int TICKET_BITS = 32;
CCF_HD unsigned long long ticket_open(int units) { return (unsigned long long)(unsigned)units << TICKET_BITS; }
CCF_HD int ticket_next(unsigned long long t) { return (int)(unsigned)t; }
CCF_HD int ticket_units(unsigned long long t) { return (int)(t >> TICKET_BITS); }

/* start of segment r of a row of R roots: the roots that CTA r of a cluster of
   csize owns in solve_kernel.  A row's blocks of roots start at these. */
CCF_HD int segment_start(int R, int csize, int r) { return (int)((long long)R * r / csize); }
constexpr int MIN_BLOCK = 64;      /* fewest roots of a unit of rows_kernel */
constexpr int NO_ROOT = 1 << 20;   /* a thread past its unit's block */
CCF_HD int row_blocks(int R, int csize, int blk)
{
	int n = 0;
	for (int r = 0; r < csize; r++) n += (segment_start(R, csize, r + 1) - segment_start(R, csize, r) + blk - 1) / blk;
	return n;
}

/* Roots per unit of a phase that evaluates n roots of each row (a step, a
   first check, an epilogue): 64, 128 or 256, the fewest that leave no more
   units than CTAs.  A unit's time is its roots' FP64 work and the chain of one
   evaluation: with two warps in a CTA instead of eight each scheduler's FP64
   pipe serves one of them, and a rectangle's off-box roots, whose star sums
   take a CTA one after another, are spread.  A row of one such unit of 256 stays
   in its CTA, which saves handing units around: up to 256 roots (full-sum
   continuation of a 60-star disc 8.0 ms, 8.6 in blocks of 64; a 60-star
   rectangle 22 in blocks of 64, 25.7 in one), 128 of a rectangle (a step of 64 roots 33 us, of 256 51; the full-sum
   continuation of 400 stars, 4 branches of 32 steps, 4.8 ms against 5.5). */
CCF_HD int block_roots(int n, int rows, int ctas, bool rectangular)
{
	if (n <= (rectangular ? NT / 2 : NT)) return NT;
	int blk = MIN_BLOCK;
	while (blk < NT && (long long)rows * ((n + blk - 1) / blk) > ctas) blk *= 2;
	return blk;
}

/* The source split of a sweep with `total` active roots, for the shortest
   sweep of a cluster of csize CTAs (solve_kernel). */
CCF_HD int source_split(int total, int csize)
{
	int S = 1, best = 1 << 30;
	for (int s2 = 1; s2 <= NT / 32; s2 *= 2)
	{
		const int nt = (total + TILE / s2 - 1) / (TILE / s2);
		const int cost = ((nt + csize - 1) / csize) * (NT / 32 + 7 * (NT / 32) / s2);
		if (cost < best)
		{
			best = cost;
			S = s2;
		}
	}
	return S;
}

/* How a sweep's sums are cut into units: tpt targets per thread, 1 where two
   would leave SMs without a unit, and 0 (one target per thread of the first
   HALF_WARPS warps only) where such units would still be no more than the SMs:
   a unit of eight warps runs two on each of the SM's four schedulers (with the
   warps that have no target kept out of the loop, the initial solve of 600
   stars in FP64 6.3 ms against 8.6, the full-sum continuation of 400 stars 4.1
   against 4.3); and
   chunks per unit, all of them where the whole sweep is less work than handing
   units around (~5 us), or where it is whole: the partial sums of its chunks
   would take more than the row's memory allows (RowsScratch), so a unit adds
   its chunks up itself, in the same order, and a row's memory stays
   proportional to its roots. */
struct SumsShape
{
	int tpt, chunks, tiles, groups, whole;
};
constexpr long long SUMS_ONE_UNIT = 1 << 16;   /* terms */
constexpr int HALF_WARPS = NT / 64;
CCF_HD SumsShape sums_shape(int total, int S, int R, int N, int nch, int rows, int sms, bool whole)
{
	SumsShape p;
	p.whole = whole ? 1 : 0;
	p.chunks = whole || (long long)total * (R + N) <= SUMS_ONE_UNIT ? nch : 1;
	p.groups = (nch + p.chunks - 1) / p.chunks;
	p.tpt = TPT;
	p.tiles = (total + TILE / S - 1) / (TILE / S);
	if ((long long)p.tiles * p.groups * rows < sms)
	{
		p.tpt = 1;
		p.tiles = (total + NT / S - 1) / (NT / S);
		if (S <= HALF_WARPS && (long long)p.tiles * p.groups * rows <= sms)
		{
			p.tpt = 0;
			p.tiles = (total + NT / 2 / S - 1) / (NT / 2 / S);
		}
	}
	return p;
}

/* whether a sweep's sums are whole: its partial sums, one per target, chunk
   and source share, take more than limit bytes */
CCF_HD bool sums_whole(int total, int S, int nch, bool mixed, long long limit)
{
	return (long long)S * total * nch * (mixed ? (long long)sizeof(float2) : (long long)sizeof(double2)) > limit;
}

/* Device memory of a launch's rows at work: of each, its partial sums (stride
   bytes), the units' shares of the next list and their lengths; slots rows at
   once, the others wait for one.  One row of a 20 000-star field has 41 MB of
   partial sums, of the 2000-star one 1.6 MB.  They grow with the square of the
   stars: a row whose sums would take more than limit bytes (from 52 000 stars
   on) has whole sums in the sweeps that exceed it, two FP64 sums per target
   and share (64 bytes a root), and its other sweeps as before.  Whole sweeps
   have fewer and longer units, which fill the GPU less evenly: the initial
   solve of 100 000 stars 159 ms, with every chunk's sums kept 149, of 200 000
   540 and 492; but such a field holds 0.6 and 0.5 GB on the device instead of
   1.5 and 4.2. */
constexpr long long ROWS_PART_BYTES = 256LL << 20;
struct RowsScratch
{
	long long stride, slots, shares, units;   /* bytes; rows; ints a slot; ints a slot */
	CCF_HD long long bytes() const { return slots * (stride + 4 * (shares + units)); }
};
/* the partial sums of one row of R roots and N stars, at most, in bytes.  S
   total is at most 10.5 tiles of the cluster with S >= 4, 2 R with S = 2
   (source_split's costs), and 8 R */
inline long long row_part_bytes(long long R, long long N, int cluster, bool mixed, long long limit)
{
	const long long chunks = (R + CHUNK - 1) / CHUNK + (N + CHUNK - 1) / CHUNK;
	const long long targets = std::min<long long>(8 * R, std::max<long long>(2 * R, 21LL * TILE * cluster / 2));
	const long long full = chunks * targets * (long long)(mixed ? sizeof(float2) : sizeof(double2));
	const long long b = full <= limit ? full : std::max<long long>(limit, 2 * targets * (long long)sizeof(double2));
	return (b + 15) / 16 * 16;
}
/* part: the largest row_part_bytes of the launch's rows, maxR: its most roots */
inline RowsScratch rows_scratch(long long part, long long maxR, long long rows)
{
	RowsScratch p;
	p.stride = part;
	/* a unit's share is 64 to 256 roots; the blocks of a row's segments may end short */
	p.shares = maxR + 17 * NT;
	p.units = maxR / MIN_BLOCK + 17;
	p.slots = 1;
	p.slots = std::max(1LL, std::min(rows, ROWS_PART_BYTES / p.bytes()));
	return p;
}

} /* namespace ccf */
