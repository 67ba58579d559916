/******************************************************************************
dfloat.cuh -- double-float arithmetic: a value is the unevaluated sum hi + lo
of two FP32 numbers with |lo| <= ulp(hi)/2, about 48 significant bits.

GB300 issues 62 FP32 FMAs for every FP64 FMA, so the critical-curve function
of the mixed-precision solver is evaluated in double-float on the FP32 pipe
instead of in FP64.  The building blocks are the classical error-free
transformations:
  two_sum       Knuth, TAOCP vol. 2, 4.2.2 (exact sum and rounding error)
  fast_two_sum  Dekker 1971 (|a| >= |b|)
  two_prod      product and its exact error from one FMA
and the double-float add / multiply / reciprocal built on them (Dekker 1971;
the same compositions as the QD library of Hida, Li and Bailey).  Every
operation uses the _rn intrinsics so the compiler cannot contract or
reassociate them.
******************************************************************************/
#pragma once

#include "common.cuh"

namespace ccf
{

struct dfl
{
	float hi, lo;
};

struct dfc   /* complex double-float */
{
	dfl re, im;
};

CCF_D dfl two_sum(float a, float b)
{
	float s = __fadd_rn(a, b);
	float v = __fsub_rn(s, a);
	float e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, v)), __fsub_rn(b, v));
	return {s, e};
}
CCF_D dfl fast_two_sum(float a, float b)
{
	float s = __fadd_rn(a, b);
	float e = __fsub_rn(b, __fsub_rn(s, a));
	return {s, e};
}
CCF_D dfl two_prod(float a, float b)
{
	float p = __fmul_rn(a, b);
	float e = __fmaf_rn(a, b, -p);
	return {p, e};
}

CCF_D dfl df_from_double(double x)
{
	float h = __double2float_rn(x);
	float l = __double2float_rn(x - (double)h);
	return {h, l};
}
CCF_D double df_to_double(dfl a) { return (double)a.hi + (double)a.lo; }
CCF_D dfl df_neg(dfl a) { return {-a.hi, -a.lo}; }

/* accurate sum (error relative to |a + b|) */
CCF_D dfl df_add(dfl a, dfl b)
{
	dfl s = two_sum(a.hi, b.hi);
	dfl t = two_sum(a.lo, b.lo);
	s.lo = __fadd_rn(s.lo, t.hi);
	s = fast_two_sum(s.hi, s.lo);
	s.lo = __fadd_rn(s.lo, t.lo);
	return fast_two_sum(s.hi, s.lo);
}
CCF_D dfl df_sub(dfl a, dfl b) { return df_add(a, df_neg(b)); }

CCF_D dfl df_mul(dfl a, dfl b)
{
	dfl p = two_prod(a.hi, b.hi);
	p.lo = __fmaf_rn(a.hi, b.lo, p.lo);
	p.lo = __fmaf_rn(a.lo, b.hi, p.lo);
	return fast_two_sum(p.hi, p.lo);
}
CCF_D dfl df_mul_f(dfl a, float b)
{
	dfl p = two_prod(a.hi, b);
	p.lo = __fmaf_rn(a.lo, b, p.lo);
	return fast_two_sum(p.hi, p.lo);
}
CCF_D dfl df_sqr(dfl a)
{
	dfl p = two_prod(a.hi, a.hi);
	p.lo = __fmaf_rn(__fmul_rn(2.0f, a.hi), a.lo, p.lo);
	return fast_two_sum(p.hi, p.lo);
}
/* sum without the low-part renormalisation: error relative to |a| + |b|,
   for accumulations whose terms do not cancel to far below their size */
CCF_D dfl df_add_fast(dfl a, dfl b)
{
	dfl s = two_sum(a.hi, b.hi);
	s.lo = __fadd_rn(s.lo, __fadd_rn(a.lo, b.lo));
	return fast_two_sum(s.hi, s.lo);
}

/* 1/a: FP32 estimate q1, residual r = 1 - a q1, one correction q1 r.  a q1
   is formed in double-float (p); p.hi lies within 2^-22 of 1, so 1 - p.hi is
   exact and r needs FP32 accuracy only (q1 r is 2^-23 of the result) */
CCF_D dfl df_rcp(dfl a)
{
	float q1 = rcp32(a.hi);
	dfl p = df_mul_f(a, q1);
	float r = __fsub_rn(__fsub_rn(1.0f, p.hi), p.lo);
	float q2 = __fmul_rn(r, q1);
	return fast_two_sum(q1, q2);
}

/* running double-float sum: the leading parts add exactly (two_sum), the low
   parts and those roundings collect in one FP32 word; dfacc_get
   renormalises.  Error ~2^-48 of the sum of |terms| */
struct dfacc
{
	float hi, lo;
};
CCF_D void dfacc_add(dfacc& a, dfl x)
{
	const dfl s = two_sum(a.hi, x.hi);
	a.hi = s.hi;
	a.lo = __fadd_rn(a.lo, __fadd_rn(s.lo, x.lo));
}
CCF_D dfl dfacc_get(dfacc a) { return fast_two_sum(a.hi, a.lo); }
/* a += x y */
CCF_D void dfacc_fma(dfacc& a, dfl x, dfl y)
{
	const float p = __fmul_rn(x.hi, y.hi);
	const float pe = __fmaf_rn(x.hi, y.hi, -p);
	const dfl s = two_sum(a.hi, p);
	a.hi = s.hi;
	a.lo = __fadd_rn(a.lo, __fadd_rn(s.lo, __fmaf_rn(x.hi, y.lo, __fmaf_rn(x.lo, y.hi, pe))));
}

/* x^2 + y^2, double-float, one renormalisation (no cancellation: error
   ~2^-47 of the result) */
CCF_D dfl df_sumsq(dfl x, dfl y)
{
	const float p = __fmul_rn(x.hi, x.hi);
	const float pe = __fmaf_rn(x.hi, x.hi, -p);
	const float q = __fmul_rn(y.hi, y.hi);
	const float qe = __fmaf_rn(y.hi, y.hi, -q);
	const dfl s = two_sum(p, q);
	const float lo = __fadd_rn(__fadd_rn(pe, qe), __fmaf_rn(__fmul_rn(2.0f, x.hi), x.lo, __fmaf_rn(__fmul_rn(2.0f, y.hi), y.lo, s.lo)));
	return fast_two_sum(s.hi, lo);
}

/* complex */
CCF_D dfc dfc_from(double2 z) { return {df_from_double(z.x), df_from_double(z.y)}; }
CCF_D double2 dfc_to(dfc a) { return make_double2(df_to_double(a.re), df_to_double(a.im)); }
CCF_D dfc dfc_add(dfc a, dfc b) { return {df_add_fast(a.re, b.re), df_add_fast(a.im, b.im)}; }
CCF_D dfc dfc_mul(dfc a, dfc b)
{
	return {df_add(df_mul(a.re, b.re), df_neg(df_mul(a.im, b.im))), df_add_fast(df_mul(a.re, b.im), df_mul(a.im, b.re))};
}
CCF_D dfc dfc_load(float4 v) { return {{v.x, v.z}, {v.y, v.w}}; }

/* x y + u z + c, real double-float, one renormalisation: the products of the
   leading parts and c's leading part sum exactly (two_prod, two_sum), every
   lower-order term collects in one FP32 sum.  Error ~2^-47 of
   |x y| + |u z| + |c| */
CCF_D dfl df_dot2_add(dfl x, dfl y, dfl u, dfl z, dfl c)
{
	const float p = __fmul_rn(x.hi, y.hi);
	const float pe = __fmaf_rn(x.hi, y.hi, -p);
	const float q = __fmul_rn(u.hi, z.hi);
	const float qe = __fmaf_rn(u.hi, z.hi, -q);
	const dfl s = two_sum(p, q);
	const dfl t = two_sum(s.hi, c.hi);
	const float e1 = __fmaf_rn(x.lo, y.hi, __fmaf_rn(x.hi, y.lo, pe));
	const float e2 = __fmaf_rn(u.lo, z.hi, __fmaf_rn(u.hi, z.lo, qe));
	const float lo = __fadd_rn(__fadd_rn(e1, e2), __fadd_rn(__fadd_rn(s.lo, t.lo), c.lo));
	return fast_two_sum(t.hi, lo);
}

/* x y + u z, real double-float, one renormalisation: error ~2^-47 of
   |x y| + |u z| */
CCF_D dfl df_dot2(dfl x, dfl y, dfl u, dfl z)
{
	const float p = __fmul_rn(x.hi, y.hi);
	const float pe = __fmaf_rn(x.hi, y.hi, -p);
	const float q = __fmul_rn(u.hi, z.hi);
	const float qe = __fmaf_rn(u.hi, z.hi, -q);
	const dfl s = two_sum(p, q);
	const float e1 = __fmaf_rn(x.lo, y.hi, __fmaf_rn(x.hi, y.lo, pe));
	const float e2 = __fmaf_rn(u.lo, z.hi, __fmaf_rn(u.hi, z.lo, qe));
	return fast_two_sum(s.hi, __fadd_rn(__fadd_rn(e1, e2), s.lo));
}

/* a b + c, complex double-float (one Horner step) */
CCF_D dfc dfc_fma(dfc a, dfc b, dfc c)
{
	return {df_dot2_add(a.re, b.re, df_neg(a.im), b.im, c.re), df_dot2_add(a.re, b.im, a.im, b.re, c.im)};
}
CCF_D float4 dfc_pack(dfc a) { return make_float4(a.re.hi, a.im.hi, a.re.lo, a.im.lo); }

/* ---------------- two double-floats per instruction ----------------

Two independent double-float chains side by side in the halves of 64-bit
register pairs, on the packed FP32 instructions (add / mul / fma .f32x2).
They run at the scalar ones' rate per operation, but one instruction carries
two: the evaluators of the tracker are held by instruction issue and fetch
(FMA pipe 41 %, issue 47 %, no_instruction the largest stall), not by the
FMA pipe, and their chains of dependent operations halve.  Every half goes
through the operations of the scalar primitive of the same name, rounded the
same way; a - b is fma(b, -1, a), the same rounding as a subtraction. */
typedef unsigned long long pk;   /* (low half, high half) */

CCF_D pk pk_make(float a, float b)
{
	pk r;
	asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
	return r;
}
CCF_D float pk_lo(pk v)
{
	float a, b;
	asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
	return a;
}
CCF_D float pk_hi(pk v)
{
	float a, b;
	asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
	return b;
}
CCF_D pk pk_add(pk a, pk b)
{
	pk r;
	asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
	return r;
}
CCF_D pk pk_mul(pk a, pk b)
{
	pk r;
	asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
	return r;
}
CCF_D pk pk_fma(pk a, pk b, pk c)
{
	pk r;
	asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
	return r;
}
CCF_D pk pk_minus_one() { return 0xbf800000bf800000ull; }
CCF_D pk pk_sub(pk a, pk b) { return pk_fma(b, pk_minus_one(), a); }
CCF_D pk pk_neg(pk a) { return pk_mul(a, pk_minus_one()); }

struct dfp   /* two double-floats */
{
	pk hi, lo;
};

CCF_D dfp dfp_make(dfl a, dfl b) { return {pk_make(a.hi, b.hi), pk_make(a.lo, b.lo)}; }
CCF_D dfl dfp_first(dfp a) { return {pk_lo(a.hi), pk_lo(a.lo)}; }
CCF_D dfl dfp_second(dfp a) { return {pk_hi(a.hi), pk_hi(a.lo)}; }
CCF_D dfp dfp_neg(dfp a) { return {pk_neg(a.hi), pk_neg(a.lo)}; }

CCF_D dfp two_sum(pk a, pk b)
{
	const pk s = pk_add(a, b);
	const pk v = pk_sub(s, a);
	return {s, pk_add(pk_sub(a, pk_sub(s, v)), pk_sub(b, v))};
}
/* a - b */
CCF_D dfp two_diff(pk a, pk b)
{
	const pk s = pk_sub(a, b);
	const pk v = pk_sub(s, a);
	return {s, pk_sub(pk_sub(a, pk_sub(s, v)), pk_add(b, v))};
}
CCF_D dfp fast_two_sum(pk a, pk b)
{
	const pk s = pk_add(a, b);
	return {s, pk_sub(b, pk_sub(s, a))};
}
/* na = -a */
CCF_D dfp fast_two_sum_neg(pk a, pk na, pk b)
{
	const pk s = pk_add(a, b);
	return {s, pk_sub(b, pk_add(s, na))};
}
CCF_D dfp dfp_sub(dfp a, dfp b)
{
	dfp s = two_diff(a.hi, b.hi);
	const dfp t = two_diff(a.lo, b.lo);
	s = fast_two_sum(s.hi, pk_add(s.lo, t.hi));
	return fast_two_sum(s.hi, pk_add(s.lo, t.lo));
}
CCF_D dfp dfp_mul(dfp a, dfp b)
{
	const pk p = pk_mul(a.hi, b.hi), np = pk_neg(p);
	pk lo = pk_fma(a.hi, b.hi, np);
	lo = pk_fma(a.hi, b.lo, lo);
	lo = pk_fma(a.lo, b.hi, lo);
	return fast_two_sum_neg(p, np, lo);
}
CCF_D dfp dfp_sumsq(dfp x, dfp y)
{
	const pk p = pk_mul(x.hi, x.hi);
	const pk pe = pk_fma(x.hi, x.hi, pk_neg(p));
	const pk q = pk_mul(y.hi, y.hi);
	const pk qe = pk_fma(y.hi, y.hi, pk_neg(q));
	const dfp s = two_sum(p, q);
	const pk lo = pk_add(pk_add(pe, qe), pk_fma(pk_add(x.hi, x.hi), x.lo, pk_fma(pk_add(y.hi, y.hi), y.lo, s.lo)));
	return fast_two_sum(s.hi, lo);
}
CCF_D dfp dfp_rcp(dfp a)
{
	const pk q1 = pk_make(rcp32(pk_lo(a.hi)), rcp32(pk_hi(a.hi)));
	const pk p = pk_mul(a.hi, q1), np = pk_neg(p);
	const pk e = pk_fma(a.lo, q1, pk_fma(a.hi, q1, np));
	const dfp t = fast_two_sum_neg(p, np, e);
	const pk r = pk_sub(pk_sub(0x3f8000003f800000ull, t.hi), t.lo);
	return fast_two_sum(q1, pk_mul(r, q1));
}
/* x^2 - y^2 (df_dot2) */
CCF_D dfp dfp_diffsq(dfp x, dfp y)
{
	const pk p = pk_mul(x.hi, x.hi);
	const pk pe = pk_fma(x.hi, x.hi, pk_neg(p));
	const pk q = pk_mul(y.hi, y.hi);
	const pk qe = pk_fma(y.hi, y.hi, pk_neg(q));
	const dfp s = two_diff(p, q);
	const pk e1 = pk_fma(x.lo, x.hi, pk_fma(x.hi, x.lo, pe));
	const pk e2 = pk_fma(y.lo, y.hi, pk_fma(y.hi, y.lo, qe));
	return fast_two_sum(s.hi, pk_add(pk_sub(e1, e2), s.lo));
}
/* a += x y: the running sums of dfacc_fma */
CCF_D void dfp_acc_fma(dfp& a, dfp x, dfp y)
{
	const pk p = pk_mul(x.hi, y.hi);
	const pk pe = pk_fma(x.hi, y.hi, pk_neg(p));
	const dfp s = two_sum(a.hi, p);
	a.hi = s.hi;
	a.lo = pk_add(a.lo, pk_add(s.lo, pk_fma(x.hi, y.lo, pk_fma(x.lo, y.hi, pe))));
}
/* the sum of the two running sums of a dfp_acc_fma accumulator */
CCF_D dfl dfp_acc_total(dfp a)
{
	const dfp t = fast_two_sum(a.hi, a.lo);
	return df_add(dfp_first(t), dfp_second(t));
}

/* x y + u z + c with -y and -z at hand (df_dot2_add): the product errors
   come out negated and save the negations of the products */
CCF_D dfp dfp_dot2_add(dfp x, dfp y, dfp ny, dfp u, dfp z, dfp nz, dfp c)
{
	const pk p = pk_mul(x.hi, y.hi);
	const pk q = pk_mul(u.hi, z.hi);
	const dfp s = two_sum(p, q);
	const dfp t = two_sum(s.hi, c.hi);
	const pk e1 = pk_fma(x.lo, ny.hi, pk_fma(x.hi, ny.lo, pk_fma(x.hi, ny.hi, p)));
	const pk e2 = pk_fma(u.lo, nz.hi, pk_fma(u.hi, nz.lo, pk_fma(u.hi, nz.hi, q)));
	return fast_two_sum(t.hi, pk_sub(pk_add(pk_add(s.lo, t.lo), c.lo), pk_add(e1, e2)));
}

/* two complex double-floats */
struct dfpc
{
	dfp re, im;
};
/* a multiplier of dfpc_fma with its negatives */
struct dfpc_mult
{
	dfp re, im, nre, nim;
};
CCF_D dfpc_mult dfpc_mult_make(dfp re, dfp im) { return {re, im, dfp_neg(re), dfp_neg(im)}; }
CCF_D dfpc dfpc_load(float4 hi, float4 lo)
{
	return {{pk_make(hi.x, hi.y), pk_make(lo.x, lo.y)}, {pk_make(hi.z, hi.w), pk_make(lo.z, lo.w)}};
}
CCF_D dfc dfpc_first(dfpc a) { return {dfp_first(a.re), dfp_first(a.im)}; }
CCF_D dfc dfpc_second(dfpc a) { return {dfp_second(a.re), dfp_second(a.im)}; }
/* a b + c (one Horner step of each half) */
CCF_D dfpc dfpc_fma(dfpc a, const dfpc_mult& b, dfpc c)
{
	return {dfp_dot2_add(a.re, b.re, b.nre, a.im, b.nim, b.im, c.re),
		dfp_dot2_add(a.re, b.im, b.nim, a.im, b.re, b.nre, c.im)};
}

} /* namespace ccf */
