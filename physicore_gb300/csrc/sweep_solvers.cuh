// sweep_solvers.cuh -- per-line tridiagonal solvers shared by the single-domain and
// batched sweeps (the reference: openmp_solver/src/diffusion_solver.cpp:116-202 and
// 390-794).
//
// FP32: forward elimination and back substitution over the whole line by one lane,
//   d_i = x_i + e_{i-1} d_{i-1}, then d_i = (b'_i c) d_{i+1} + b'_i d_i downwards
// (both from a zero carry; b' as a pair hi + lo).  These sweeps move their bytes at
// the copy bandwidth; what a shorter chain would save they do not wait for.
//
// FP64: the FP64 pipe sets the pace (one warp instruction per 20 cycles of an SM, with
// a latency of several of those), so the line is solved with the fewest
// operations and in two halves side by side.  It is eliminated from both ends
// towards a meeting point and solved outwards from there (a twisted factorisation of
// the same matrix); the halves belong to the CTA's two warps.  With r = dt D / h^2,
// b'_j and e_j = r b'_j the reference's own values (the matrix reads the same from
// either end, so both halves use one table), each half runs
//   inward    d_j = x_j + e_{j-1} d_{j-1}                j = 0 .. L-1
//   meeting   y   = w d + w' d'                          (d' the other half's last d)
//   outward   y_j = d_j + e_{j+1} y_{j+1}                j = L-2 .. 0
// and the line's solution is b'_j y_j.  That factor depends on the substrate and the
// position along the swept axis only, so it commutes with the sweeps of the other
// axes: a step's sweeps leave it out and the last one multiplies by the product
// (SC = 1): 7 FP64 operations per point and 3-D step instead of 9 (8 at the head
// points, whose factor is formed per point), and 1 in the dependent chain of a point
// instead of 3.  A mesh whose factors would let the values
// between the sweeps grow past 2^20 of the field's applies them in every sweep.
// 160x144x128, 3 substrates: x 97 -> 58, y 86 -> 56, z 80 -> 75 us.
#pragma once

#include "pcg_internal.cuh"

namespace pcg {
namespace solvers {

constexpr int kBlock = 8; // recurrence steps per pipelined block

// Threads of a sweep CTA: a warp per tile (FP32), or one for each half of its lines.
// FP64 kernels are compiled for 8 CTAs an SM (128 registers), 16 warps: with the 168 of
// 6 CTAs, 64^3 x 8, 1024 tiles, took 24, 24 and 36 us for x, y and z instead of 19, 19 and 27.
// FP32 kernels state no number (0): stating one CTA gave them 150 to 196 registers instead of
// 108 to 120, and 97x131x61 x 5 took 40.9 instead of 34.6 us a step.
template <typename T>
constexpr int sweep_threads()
{
	return sizeof(T) == 4 ? 32 : 64;
}

// Points of a line that the first warp solves: all (FP32), or a whole number of
// blocks near the middle; lines of at most one block have no second half.
template <typename T>
__host__ __device__ constexpr uint32_t line_split(uint32_t n)
{
	return sizeof(T) == 4 || n <= 8 ? n : (n + 8) / 16 * 8;
}

// Mass-check accumulators: a lane's running total of the values a sweep reads
// (before the step's first sweep) or writes (after its last sweep), fused into
// the solvers so the check needs no pass of its own.  FP32: a float pair
// hi + lo accumulated with Knuth's TwoSum (error-free), fed with FP32 sums of
// blocks of points, so about one extra instruction per point; FP64: a double.
template <typename T>
struct MassAcc;

template <>
struct MassAcc<float>
{
	float hi, lo;
	__device__ __forceinline__ void zero() { hi = lo = 0.f; }
	__device__ __forceinline__ void add(float x)
	{
		const float s = __fadd_rn(hi, x);
		const float bb = __fsub_rn(s, hi);
		lo = __fadd_rn(lo, __fadd_rn(__fsub_rn(hi, __fsub_rn(s, bb)), __fsub_rn(x, bb)));
		hi = s;
	}
	template <int P>
	__device__ __forceinline__ void add_block(const float (&x)[P])
	{
		static_assert(P == 8, "blocks of 8 points");
		add(__fadd_rn(__fadd_rn(__fadd_rn(x[0], x[1]), __fadd_rn(x[2], x[3])),
					  __fadd_rn(__fadd_rn(x[4], x[5]), __fadd_rn(x[6], x[7]))));
	}
	__device__ __forceinline__ double value() const { return (double)hi + (double)lo; }
};

template <>
struct MassAcc<double>
{
	double v;
	__device__ __forceinline__ void zero() { v = 0.0; }
	__device__ __forceinline__ void add(double x) { v += x; }
	template <int P>
	__device__ __forceinline__ void add_block(const double (&x)[P])
	{
		static_assert(P == 8, "blocks of 8 points");
		v += ((x[0] + x[1]) + (x[2] + x[3])) + ((x[4] + x[5]) + (x[6] + x[7]));
	}
	__device__ __forceinline__ double value() const { return v; }
};

// Mass-check modes of a solver call (bits): sum the inputs, sum the outputs.
enum : int
{
	kMcIn = 1,
	kMcOut = 2,
};

// Adds the totals v of the first `width` lanes of the warp to FP64 totals with
// atomics, where lanes l and l + stride (stride <= 32) add to the same total: the
// classes are summed by a tree over strides stride, 2*stride, ..., then lane
// l < stride adds its class's sum to *dst (its own target).  All `width` lanes
// of the warp call it.
__device__ __forceinline__ void flush_classes(double v, uint32_t stride, uint32_t width, double* dst)
{
	const uint32_t lane = threadIdx.x & 31;
	const uint32_t mask = width >= 32 ? 0xffffffffu : ((1u << width) - 1u);
	for (uint32_t k = stride; k < 32; k <<= 1)
	{
		const double t = __shfl_down_sync(mask, v, k);
		if (lane + k < width)
			v += t;
	}
	if (lane < stride && lane < width && v != 0.0)
		atomicAdd(dst, v);
}

// Points of one line in shared memory, counted from the end where a warp starts:
// point j at p[DIR * j * stride].  STRIDE 0: the run-time stride.
template <typename T, int STRIDE, int DIR>
struct Strided
{
	T* p;
	uint32_t st;
	__device__ __forceinline__ int stride() const { return DIR * (STRIDE ? STRIDE : (int)st); }
	__device__ __forceinline__ T& at(uint32_t j) const { return p[(int)j * stride()]; }
	__device__ __forceinline__ void load(uint32_t j, T (&x)[kBlock]) const
	{
		const T* b = p + (int)j * stride();
#pragma unroll
		for (int k = 0; k < kBlock; k++)
			x[k] = b[k * stride()];
	}
	__device__ __forceinline__ void store(uint32_t j, const T (&x)[kBlock]) const
	{
		T* b = p + (int)j * stride();
#pragma unroll
		for (int k = 0; k < kBlock; k++)
			b[k * stride()] = x[k];
	}
};

// FP32 points side by side (one substrate, a lane per row): blocks move as two
// 16-byte accesses, so the rows of a warp, an odd number of 16-byte chunks apart, meet
// no bank conflict.  Rows start on 16-byte boundaries and blocks at multiples of 8.
struct RowLine
{
	float* p;
	__device__ __forceinline__ float& at(uint32_t j) const { return p[j]; }
	__device__ __forceinline__ void load(uint32_t j, float (&x)[kBlock]) const
	{
#pragma unroll
		for (int c = 0; c < 2; c++)
		{
			const float4 v = *reinterpret_cast<const float4*>(p + j + 4 * c);
			x[4 * c] = v.x, x[4 * c + 1] = v.y, x[4 * c + 2] = v.z, x[4 * c + 3] = v.w;
		}
	}
	__device__ __forceinline__ void store(uint32_t j, const float (&x)[kBlock]) const
	{
#pragma unroll
		for (int c = 0; c < 2; c++)
			*reinterpret_cast<float4*>(p + j + 4 * c) = make_float4(x[4 * c], x[4 * c + 1], x[4 * c + 2], x[4 * c + 3]);
	}
};

template <typename T>
struct LineCoef;

// The scale factors of one lane's half line at the last FP64 sweep: g the column's
// factor from the other axes, mid = g times the line's converged factor (the head
// points' are in LineCoef).
template <typename T>
struct LineScale
{
	double g, mid;
	bool on; // false: g and mid are 1 and the line's own factors are left out
};

// ------------------------------------------------------------------ FP32

// One lane's coefficients along a line, from the axis's table: points j < H read the
// substrate's head rows, points H <= j < n-1 share the middle constants, and point
// n-1 has its own (when H >= n the head holds the whole line).  H is a multiple of
// kBlock, so a block of points is either all head or all middle/last.
template <>
struct LineCoef<float>
{
	const float* hB;
	const float* hE;
	const float* hBl; // lo parts of the multipliers (head rows)
	uint32_t H, n;
	float mB, mE, lB, lE, c;
	float mBl, lBl; // lo parts of the middle and last multipliers
};

// FP32 table of an axis: [head b' (S x H) | head e (S x H) | mid b' | mid e |
// last b' | last e | c], the five constant arrays kS = S rounded up to 16 bytes long,
// then [head b' lo (S x H) | mid b' lo | last b' lo].
__device__ __forceinline__ LineCoef<float> line_coef(const float* tab, uint32_t S, uint32_t H, uint32_t n, uint32_t s,
													 uint32_t)
{
	const uint32_t kS = (S + 3) / 4 * 4;
	const float* k = tab + 2ull * S * H;
	const float* lo = k + 5 * kS;
	LineCoef<float> L;
	L.hB = tab + (uint64_t)s * H;
	L.hE = tab + (uint64_t)S * H + (uint64_t)s * H;
	L.H = H;
	L.n = n;
	L.mB = __ldg(k + s);
	L.mE = __ldg(k + kS + s);
	L.lB = __ldg(k + 2 * kS + s);
	L.lE = __ldg(k + 3 * kS + s);
	L.c = __ldg(k + 4 * kS + s);
	L.hBl = lo + (uint64_t)s * H;
	L.mBl = __ldg(lo + (uint64_t)S * H + s);
	L.lBl = __ldg(lo + (uint64_t)S * H + kS + s);
	return L;
}

// One backward step d = (x + c d) b', evaluated as (b' c) d + b' x with the coupling
// b' c = RN(bh * c) and the product b' x taken with the multiplier's pair bh + bl
// (the host's column-sum-exact multipliers account for the coupling's rounding), so
// the chain from one point to the next is a single fma.
__device__ __forceinline__ float bwd_step(float c, float d, float x, float bh, float bl)
{
	const float bc = bh * c;
	const float xb = dev::fmadd(x, bh, x * bl);
	return dev::fmadd(bc, d, xb);
}

__device__ __forceinline__ float coef_at(const float* head, uint32_t H, float mid, float last, uint32_t n, uint32_t j)
{
	return j < H ? __ldg(head + j) : (j == n - 1 ? last : mid);
}

// One line of n points in shared memory with the lane's coefficients L.  The line is
// three runs: head blocks of kBlock points [0, hb) (coefficients from the head
// rows), middle blocks [hb, q) (the middle constants, held in registers) and the
// points from q * kBlock on, which hold point n-1 (coefficients chosen per point;
// at most 2 kBlock - 1 of them).  Within a run the next block's points (and head
// coefficients) are requested before the current block's dependent chain, so
// their latency overlaps it; the middle run, nearly the whole line, alternates two
// register sets, so that its blocks carry no copies or tests.  Which run a block
// is in is the same for every lane of a warp (one n and H per launch).
//
// SMALL keeps the loops rolled: the batched y and z, with more code around the
// solver, waited on instruction fetches with the compiler's own unrolling (990 served
// requests: y 8.87 -> 8.52, z 9.09 -> 8.81 ms; 256 domains 2.29 -> 2.22 ms a step).  One
// domain's kernels keep the unrolling, which long lines gain from (30,000 x 1: 340
// instead of 364 us).
//
// MC (kMcIn / kMcOut bits) adds the line's input values to *acc_in and its
// solved values to *acc_out.
template <class AC, int MC, bool SMALL>
__device__ __forceinline__ void solve_line(const AC& ac, uint32_t n, const LineCoef<float>& L, MassAcc<float>* acc_in,
										   MassAcc<float>* acc_out)
{
	constexpr int P = kBlock, NV = P / 4;
	const uint32_t nb = n / P;
	const uint32_t hb = min(L.H / P, nb);
	const uint32_t q = max((n - 1) / P, hb); // blocks [hb, q) have j0 >= H and j0 + P <= n - 1
	const float c = L.c;
	// the middle coupling of the backward step, as bwd_step forms it per point
	const float mbc = L.mB * c;
	auto fetch_head = [&](const float* head, uint32_t b, float(&out)[P]) {
#pragma unroll
		for (int v = 0; v < NV; v++)
		{
			const float4 q = __ldg(reinterpret_cast<const float4*>(head + b * P) + v);
			out[4 * v] = q.x, out[4 * v + 1] = q.y, out[4 * v + 2] = q.z, out[4 * v + 3] = q.w;
		}
	};
	float d = 0.f;

	// ---- forward elimination
	auto fwd_mid = [&](uint32_t b, float(&x)[P]) {
		if constexpr ((MC & kMcIn) != 0)
			acc_in->add_block(x);
#pragma unroll
		for (int k = 0; k < P; k++)
			x[k] = d = dev::fmadd(L.mE, d, x[k]);
		ac.store(b * P, x);
	};
	if (hb)
	{
		float x[P], xn[P];
		float e[P], en[P];
		ac.load((0) * P, x);
		fetch_head(L.hE, 0, e);
		auto fwd_head = [&](uint32_t b) {
			if (b + 1 < hb)
			{
				ac.load((b + 1) * P, xn);
				fetch_head(L.hE, b + 1, en);
			}
			if constexpr ((MC & kMcIn) != 0)
				acc_in->add_block(x);
#pragma unroll
			for (int k = 0; k < P; k++)
				x[k] = d = dev::fmadd(e[k], d, x[k]);
			ac.store(b * P, x);
#pragma unroll
			for (int k = 0; k < P; k++)
			{
				x[k] = xn[k];
				e[k] = en[k];
			}
		};
		if constexpr (SMALL)
		{
#pragma unroll 1
			for (uint32_t b = 0; b < hb; b++)
				fwd_head(b);
		}
		else
			for (uint32_t b = 0; b < hb; b++)
				fwd_head(b);
	}
	if (hb < q)
	{
		float xa[P], xb[P];
		uint32_t b = hb;
		ac.load((b) * P, xa);
		auto fwd_two = [&](uint32_t b) {
			ac.load((b + 1) * P, xb);
			fwd_mid(b, xa);
			ac.load((b + 2) * P, xa);
			fwd_mid(b + 1, xb);
		};
		if constexpr (SMALL)
		{
#pragma unroll 1
			for (; b + 2 < q; b += 2)
				fwd_two(b);
		}
		else
			for (; b + 2 < q; b += 2)
				fwd_two(b);
		if (b + 1 < q)
		{
			ac.load((b + 1) * P, xb);
			fwd_mid(b, xa);
			fwd_mid(b + 1, xb);
		}
		else
			fwd_mid(b, xa);
	}
	auto fwd_last = [&](uint32_t j) {
		const float xj = ac.at(j);
		if constexpr ((MC & kMcIn) != 0)
			acc_in->add(xj);
		d = dev::fmadd(coef_at(L.hE, L.H, L.mE, L.lE, n, j), d, xj);
		ac.at(j) = d;
	};
	if constexpr (SMALL)
	{
#pragma unroll 1
		for (uint32_t j = q * P; j < n; j++)
			fwd_last(j);
	}
	else
		for (uint32_t j = q * P; j < n; j++)
			fwd_last(j);

	// ---- back substitution
	d = 0.f;
	auto bwd_last = [&](uint32_t j) {
		const float bl = coef_at(L.hBl, L.H, L.mBl, L.lBl, n, j);
		d = bwd_step(c, d, ac.at(j), coef_at(L.hB, L.H, L.mB, L.lB, n, j), bl);
		ac.at(j) = d;
		if constexpr ((MC & kMcOut) != 0)
			acc_out->add(d);
	};
	if constexpr (SMALL)
	{
#pragma unroll 1
		for (uint32_t j = n; j-- > q * P;)
			bwd_last(j);
	}
	else
		for (uint32_t j = n; j-- > q * P;)
			bwd_last(j);
	auto bwd_mid = [&](uint32_t b, float(&x)[P]) {
#pragma unroll
		for (int k = P - 1; k >= 0; k--)
			x[k] = d = dev::fmadd(mbc, d, dev::fmadd(x[k], L.mB, x[k] * L.mBl));
		if constexpr ((MC & kMcOut) != 0)
			acc_out->add_block(x);
		ac.store(b * P, x);
	};
	if (hb < q)
	{
		float xa[P], xb[P];
		uint32_t b = q - 1;
		ac.load((b) * P, xa);
		auto bwd_two = [&](uint32_t b) {
			ac.load((b - 1) * P, xb);
			bwd_mid(b, xa);
			ac.load((b - 2) * P, xa);
			bwd_mid(b - 1, xb);
		};
		if constexpr (SMALL)
		{
#pragma unroll 1
			for (; b >= hb + 2; b -= 2)
				bwd_two(b);
		}
		else
			for (; b >= hb + 2; b -= 2)
				bwd_two(b);
		if (b >= hb + 1)
		{
			ac.load((b - 1) * P, xb);
			bwd_mid(b, xa);
			bwd_mid(b - 1, xb);
		}
		else
			bwd_mid(b, xa);
	}
	if (hb)
	{
		float x[P], xn[P];
		float bb[P], bn[P], bl[P], bln[P];
		ac.load((hb - 1) * P, x);
		fetch_head(L.hB, hb - 1, bb);
		fetch_head(L.hBl, hb - 1, bl);
		auto bwd_head = [&](uint32_t b) {
			if (b > 0)
			{
				ac.load((b - 1) * P, xn);
				fetch_head(L.hB, b - 1, bn);
				fetch_head(L.hBl, b - 1, bln);
			}
#pragma unroll
			for (int k = P - 1; k >= 0; k--)
				x[k] = d = bwd_step(c, d, x[k], bb[k], bl[k]);
			if constexpr ((MC & kMcOut) != 0)
				acc_out->add_block(x);
			ac.store(b * P, x);
#pragma unroll
			for (int k = 0; k < P; k++)
			{
				x[k] = xn[k];
				bb[k] = bn[k];
				bl[k] = bln[k];
			}
		};
		if constexpr (SMALL)
		{
#pragma unroll 1
			for (uint32_t b = hb; b-- > 0;)
				bwd_head(b);
		}
		else
			for (uint32_t b = hb; b-- > 0;)
				bwd_head(b);
	}
}

// ------------------------------------------------------------------ FP64

// One lane's coefficients for its half of a line, from the axis's table (capi.cu):
// points j < H take theirs from the substrate's head rows, the others share e.
template <>
struct LineCoef<double>
{
	const double* hE; // inward coefficients of the head points
	const double* hG; // outward
	const double* hF; // scale factors
	uint32_t H;
	double e;
	double ws, wo; // meeting point: weights of the half's own and the other half's value
};

__device__ __forceinline__ LineCoef<double> line_coef(const double* tab, uint32_t S, uint32_t H, uint32_t, uint32_t s,
													  uint32_t half)
{
	const double* k = tab + 3 * S * H + s;
	LineCoef<double> L;
	L.hE = tab + s * H;
	L.hG = tab + (S + s) * H;
	L.hF = tab + (2 * S + s) * H;
	L.H = H;
	L.e = __ldg(k);
	L.ws = __ldg(k + S);
	L.wo = __ldg(k + (2 + half) * S);
	return L;
}

// The 8 head coefficients from point j on.
__device__ __forceinline__ void head_block(const double* row, uint32_t j, double (&c)[kBlock])
{
#pragma unroll
	for (int v = 0; v < kBlock / 2; v++)
	{
		const double2 a = __ldg(reinterpret_cast<const double2*>(row + j) + v);
		c[2 * v] = a.x, c[2 * v + 1] = a.y;
	}
}

// Inward elimination of a half line of len points; returns the last value (also
// left in the tile).  The blocks of 8 that hold head points take their
// coefficients from the head rows; the others alternate two register sets, the
// next block's points requested before the current block's dependent chain.  All
// counts are the same for every lane of a warp.
template <class AC, int MC>
__device__ __forceinline__ double solve_inward(const AC& ac, uint32_t len, const LineCoef<double>& L, MassAcc<double>* acc)
{
	constexpr int P = kBlock;
	const uint32_t nb = len / P, hb = min(L.H / P, nb);
	double d = 0.0;
	auto mid = [&](uint32_t b, double(&x)[P]) {
		if constexpr ((MC & kMcIn) != 0)
			acc->add_block(x);
#pragma unroll
		for (int k = 0; k < P; k++)
			x[k] = d = dev::fmadd(L.e, d, x[k]);
		ac.store(b * P, x);
	};
	if (hb)
	{
		double x[P], xn[P], c[P], cn[P];
		ac.load(0, x);
		head_block(L.hE, 0, c);
#pragma unroll 1
		for (uint32_t b = 0; b < hb; b++)
		{
			if (b + 1 < hb)
			{
				ac.load((b + 1) * P, xn);
				head_block(L.hE, (b + 1) * P, cn);
			}
			if constexpr ((MC & kMcIn) != 0)
				acc->add_block(x);
#pragma unroll
			for (int k = 0; k < P; k++)
				x[k] = d = dev::fmadd(c[k], d, x[k]);
			ac.store(b * P, x);
#pragma unroll
			for (int k = 0; k < P; k++)
			{
				x[k] = xn[k];
				c[k] = cn[k];
			}
		}
	}
	if (hb < nb)
	{
		double xa[P], xb[P];
		uint32_t b = hb;
		ac.load(b * P, xa);
		for (; b + 2 < nb; b += 2)
		{
			ac.load((b + 1) * P, xb);
			mid(b, xa);
			ac.load((b + 2) * P, xa);
			mid(b + 1, xb);
		}
		if (b + 1 < nb)
		{
			ac.load((b + 1) * P, xb);
			mid(b, xa);
			mid(b + 1, xb);
		}
		else
			mid(b, xa);
	}
	for (uint32_t j = nb * P; j < len; j++)
	{
		const double x = ac.at(j);
		if constexpr ((MC & kMcIn) != 0)
			acc->add(x);
		d = dev::fmadd(j < L.H ? __ldg(L.hE + j) : L.e, d, x);
		ac.at(j) = d;
	}
	return d;
}

// Outward substitution from the meeting point's value y.  SC: the stored values
// are the solution (times the column's factor), else the solution over the line's
// factors.
template <class AC, int MC, int SC>
__device__ __forceinline__ void solve_outward(const AC& ac, uint32_t len, const LineCoef<double>& L, double ymeet,
											  const LineScale<double>& F, MassAcc<double>* acc)
{
	constexpr int P = kBlock;
	const uint32_t nb = len / P, hb = min(L.H / P, nb);
	ac.at(len - 1) = ymeet; // the recurrence then starts from a zero carry
	double y = 0.0;
	auto mid = [&](uint32_t b, double(&x)[P]) {
#pragma unroll
		for (int k = P - 1; k >= 0; k--)
		{
			y = dev::fmadd(L.e, y, x[k]);
			x[k] = SC ? y * F.mid : y;
		}
		if constexpr ((MC & kMcOut) != 0)
			acc->add_block(x);
		ac.store(b * P, x);
	};
	for (int j = (int)len - 1; j >= (int)(nb * P); j--)
	{
		y = dev::fmadd((uint32_t)j < L.H ? __ldg(L.hG + j) : L.e, y, ac.at(j));
		const double o = SC ? y * ((uint32_t)j < L.H ? (F.on ? F.g * __ldg(L.hF + j) : 1.0) : F.mid) : y;
		ac.at(j) = o;
		if constexpr ((MC & kMcOut) != 0)
			acc->add(o);
	}
	if (hb < nb)
	{
		double xa[P], xb[P];
		uint32_t b = nb - 1;
		ac.load(b * P, xa);
		for (; b >= hb + 2; b -= 2)
		{
			ac.load((b - 1) * P, xb);
			mid(b, xa);
			ac.load((b - 2) * P, xa);
			mid(b - 1, xb);
		}
		if (b >= hb + 1)
		{
			ac.load((b - 1) * P, xb);
			mid(b, xa);
			mid(b - 1, xb);
		}
		else
			mid(b, xa);
	}
#pragma unroll 1
	for (int b = (int)hb - 1; b >= 0; b--)
	{
		double x[P], c[P], f[P];
		ac.load((uint32_t)b * P, x);
		head_block(L.hG, (uint32_t)b * P, c);
		if constexpr (SC != 0)
			head_block(L.hF, (uint32_t)b * P, f);
#pragma unroll
		for (int k = P - 1; k >= 0; k--)
		{
			y = dev::fmadd(c[k], y, x[k]);
			x[k] = SC ? y * (F.on ? F.g * f[k] : 1.0) : y;
		}
		if constexpr ((MC & kMcOut) != 0)
			acc->add_block(x);
		ac.store((uint32_t)b * P, x);
	}
}

// ------------------------------------------------------------------ tiles

// The lines of one tile, one per lane: `left` reaches a lane's line from point 0,
// `right` from point n-1.  Lanes without a line (on == false) only take part in the
// barriers.  FP32: the CTA's one warp solves whole lines.  FP64: warp `half` solves
// its half of them; two barriers separate the reads of the other half's meeting
// value from the writes around them (a line without a second half needs none).
template <typename T, class ACL, class ACR, int MC, int SC, bool SMALL = false>
__device__ __forceinline__ void solve_tile(const ACL& left, const ACR& right, uint32_t n, uint32_t half, bool on,
										   const LineCoef<T>& L, const LineScale<T>& F, MassAcc<T>* acc_in = nullptr,
										   MassAcc<T>* acc_out = nullptr)
{
	if constexpr (sizeof(T) == 4)
	{
		if (on)
			solve_line<ACL, MC, SMALL>(left, n, L, acc_in, acc_out);
	}
	else
	{
		const uint32_t m = line_split<T>(n);
		T own = T(0), other = T(0);
		if (on)
		{
			if (half == 0)
				own = solve_inward<ACL, MC>(left, m, L, acc_in);
			else if (n > m)
				own = solve_inward<ACR, MC>(right, n - m, L, acc_in);
		}
		if (n > m)
		{
			__syncthreads();
			if (on)
				other = half == 0 ? right.at(n - m - 1) : left.at(m - 1);
			__syncthreads();
		}
		if (on)
		{
			// the solution at the half's inner end, over its scale factor
			const T y = dev::fmadd(L.ws, own, L.wo * other);
			if (half == 0)
				solve_outward<ACL, MC, SC>(left, m, L, y, F, acc_out);
			else if (n > m)
				solve_outward<ACR, MC, SC>(right, n - m, L, y, F, acc_out);
		}
	}
}

} // namespace solvers
} // namespace pcg
