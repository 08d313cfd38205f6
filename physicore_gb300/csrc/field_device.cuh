// field_device.cuh -- per-item device code of the Dirichlet and bulk phases,
// shared by the single-domain kernels (field_ops.cu) and the batched ones (batch.cu).
//
// Dirichlet (openmp_solver/src/dirichlet_solver.cpp:22-93): the reference writes
// the x-min, x-max, y-min, y-max, z-min, z-max faces one after another (a later
// face wins on shared edges) and then the interior voxels.  A face item is one
// (face voxel, substrate); it applies the face of highest precedence whose
// condition holds, so edges resolve exactly as the sequential order does.
//
// Bulk (openmp_solver/src/bulk_solver.cpp:12-49): D = (D + dt*S*T)/(1 + dt*(U+S)).
#pragma once

#include "pcg_internal.cuh"

namespace pcg {

struct FaceArgs
{
	void* field;
	const void* values; // real [6*S]: face f = axis*2 + side
	const uint8_t* conds;
	uint32_t face_mask; // bit f set when face f exists
	uint64_t S, nx, ny, nz, pitch;
	uint64_t cnt_x, cnt_y, cnt_z; // voxels on each pair of faces
	uint64_t total;               // face voxels (all pairs)
};

// Fills the face geometry of a mesh from its per-face presence.
inline FaceArgs make_face_args(const Context* c)
{
	FaceArgs a {};
	uint32_t mask = 0;
	for (int axis = 0; axis < c->dims; axis++)
		for (int side = 0; side < 2; side++)
			if (c->face_on[axis][side])
				mask |= 1u << (axis * 2 + side);
	const uint64_t nx = c->n[0], ny = c->n[1], nz = c->n[2];
	a.field = c->field.ptr;
	a.values = c->face_values.ptr;
	a.conds = static_cast<const uint8_t*>(c->face_conds.ptr);
	a.face_mask = mask;
	a.S = c->S;
	a.nx = nx, a.ny = ny, a.nz = nz;
	a.pitch = c->pitch;
	a.cnt_x = (mask & 0x3) ? 2 * ny * nz : 0;
	a.cnt_y = (mask & 0xc) ? 2 * nx * nz : 0;
	a.cnt_z = (mask & 0x30) ? 2 * nx * ny : 0;
	a.total = a.cnt_x + a.cnt_y + a.cnt_z;
	return a;
}

#ifdef __CUDACC__
namespace fielddev {

// Face item idx < total*S.
template <typename T>
__device__ __forceinline__ void face_item(const FaceArgs& a, uint64_t idx)
{
	const T* vals = static_cast<const T*>(a.values);
	T* f = static_cast<T*>(a.field);
	const uint64_t s = idx % a.S;
	uint64_t k = idx / a.S;
	uint64_t x, y, z;
	if (k < a.cnt_x)
	{ // x faces: k -> (side, y, z)
		const uint64_t per = a.ny * a.nz;
		x = (k / per) ? a.nx - 1 : 0;
		y = (k % per) % a.ny;
		z = (k % per) / a.ny;
	}
	else if ((k -= a.cnt_x) < a.cnt_y)
	{
		const uint64_t per = a.nx * a.nz;
		y = (k / per) ? a.ny - 1 : 0;
		x = (k % per) % a.nx;
		z = (k % per) / a.nx;
	}
	else
	{
		k -= a.cnt_y;
		const uint64_t per = a.nx * a.ny;
		z = (k / per) ? a.nz - 1 : 0;
		x = (k % per) % a.nx;
		y = (k % per) / a.nx;
	}
	// precedence: the reference applies faces 0..5 in order, so scan 5..0
	const uint64_t coord[3] = { x, y, z };
	const uint64_t last[3] = { a.nx - 1, a.ny - 1, a.nz - 1 };
	for (int fi = 5; fi >= 0; fi--)
	{
		if (!(a.face_mask & (1u << fi)))
			continue;
		const int axis = fi >> 1, side = fi & 1;
		if (coord[axis] != (side ? last[axis] : 0))
			continue;
		if (a.conds[fi * a.S + s])
		{
			f[(z * a.ny + y) * a.pitch + x * a.S + s] = vals[fi * a.S + s];
			break;
		}
	}
}

// The bulk update of one voxel-substrate (bulk_solver.cpp:12-49): D' = (D + dt S T) /
// (1 + dt (U + S)); FP32 as D + (dt S T - D dt (U + S)) / (1 + dt (U + S)), so that a
// small dt (U + S) keeps its precision (its sum with 1 only scales the correction).
template <typename T>
__device__ __forceinline__ T bulk_value(T D, T Sr, T U, T Tt, T dt)
{
	if constexpr (sizeof(T) == 4)
	{
		const T a = dt * Sr * Tt, b = dt * (U + Sr);
		return D + fmaf(-D, b, a) / (T(1) + b);
	}
	else
		// fused by name: where the products are hoisted out of a loop the compiler would not
		return fma(dt * Sr, Tt, D) / fma(dt, U + Sr, T(1));
}

// The 16-byte chunk c of row r (fields and per-voxel tables have the same layout, and
// rows start on 32-byte boundaries; the row's last chunk may hold fewer of its
// elements).  Memory sets the pace only with whole chunks in flight per thread: one
// element per thread and turn, a warp walking a row, ran at 0.5 TB/s.
template <typename T, bool PER_VOXEL>
__device__ __forceinline__ void bulk_chunk(T* field, const T* supply, const T* uptake, const T* target, uint32_t row_len,
										   uint64_t pitch, uint64_t r, uint32_t c, uint32_t S, T dt)
{
	constexpr uint32_t VN = 16 / sizeof(T);
	union Chunk
	{
		uint4 u;
		T t[VN];
	};
	const uint64_t off = r * pitch + (uint64_t)c * VN;
	const uint32_t left = row_len - c * VN;
	Chunk d, sp, up, tp;
	d.u = *reinterpret_cast<const uint4*>(field + off);
	if constexpr (PER_VOXEL)
	{
		sp.u = __ldg(reinterpret_cast<const uint4*>(supply + off));
		up.u = __ldg(reinterpret_cast<const uint4*>(uptake + off));
		tp.u = __ldg(reinterpret_cast<const uint4*>(target + off));
	}
	else
	{
		uint32_t s = c * VN % S;
#pragma unroll
		for (uint32_t q = 0; q < VN; q++)
		{
			sp.t[q] = __ldg(supply + s);
			up.t[q] = __ldg(uptake + s);
			tp.t[q] = __ldg(target + s);
			if (++s == S)
				s = 0;
		}
	}
#pragma unroll
	for (uint32_t q = 0; q < VN; q++)
		d.t[q] = bulk_value(d.t[q], sp.t[q], up.t[q], tp.t[q], dt);
	if (left >= VN)
		*reinterpret_cast<uint4*>(field + off) = d.u;
	else // the padding after the row keeps its zeros
		for (uint32_t q = 0; q < left; q++)
			field[off + q] = d.t[q];
}

// The boundary faces of the voxels of one half of a solved y/z column in shared
// memory (the last sweep of the step, so these are the values the reference's
// Dirichlet pass would write next).  The column is substrate s of voxel x of a row
// at all points of the swept axis; `col` is the half's lowest point, its `len`
// points `stride` apart; `first` / `last` tell whether it holds the line's end
// points; `o` is the index along the third axis.  Faces apply in the reference's
// order x-min, x-max, y-min, y-max, z-min, z-max, a later face winning: first the
// faces whose plane holds the whole column, then the two faces of the swept axis at
// its ends.  ARGS: face_values, face_conds, face_mask, S, nx, ny, nz.
template <typename T, int AXIS, typename ARGS>
__device__ __forceinline__ void faces_on_half(const ARGS& f, uint32_t x, uint32_t s, uint32_t o, T* col, uint32_t len,
											  uint32_t stride, bool first, bool last)
{
	const T* vals = static_cast<const T*>(f.face_values);
	const uint32_t S = (uint32_t)f.S;
	bool has = false;
	T v = T(0);
	auto take = [&](uint32_t fi) {
		if (((f.face_mask >> fi) & 1u) && f.face_conds[fi * S + s])
		{
			v = vals[fi * S + s];
			has = true;
		}
	};
	if (x == 0)
		take(0);
	if (x == f.nx - 1)
		take(1);
	const uint32_t n_other = (uint32_t)(AXIS == 2 ? f.ny : f.nz); // the axis that is neither x nor swept
	const uint32_t f_other = AXIS == 2 ? 2 : 4;
	if (o == 0)
		take(f_other);
	if (o == n_other - 1)
		take(f_other + 1);
	if (has)
		for (uint32_t j = 0; j < len; j++)
			col[j * stride] = v;
	const uint32_t f_swept = AXIS == 2 ? 4 : 2;
	if (first && ((f.face_mask >> f_swept) & 1u) && f.face_conds[f_swept * S + s])
		col[0] = vals[f_swept * S + s];
	if (last && ((f.face_mask >> (f_swept + 1)) & 1u) && f.face_conds[(f_swept + 1) * S + s])
		col[(len - 1) * stride] = vals[(f_swept + 1) * S + s];
}

// The bulk update, with uniform rates, of `len` points of substrate s of a column in
// shared memory, `stride` apart.
template <typename T>
__device__ __forceinline__ void bulk_on_half(const void* const* tables, T dt, uint32_t s, T* col, uint32_t len,
											 uint32_t stride)
{
	const T Sr = __ldg(static_cast<const T*>(tables[0]) + s), U = __ldg(static_cast<const T*>(tables[1]) + s),
			Tt = __ldg(static_cast<const T*>(tables[2]) + s);
#pragma unroll 4
	for (uint32_t j = 0; j < len; j++)
		col[j * stride] = bulk_value(col[j * stride], Sr, U, Tt, dt);
}

} // namespace fielddev
#endif

} // namespace pcg
