// sweeps.cu -- ADI/LOD tridiagonal sweeps along x, y and z on sm_103a.
//
// Each line solves the reference's matrix of its substrate (openmp_solver/src/
// diffusion_solver.cpp:116-202 for x, 390-794 for y/z; coefficients of
// diffusion_solver.cpp:29-86); the solvers are in sweep_solvers.cuh.
//
// GB300 mapping (our own design):
//  * A line must stay on chip between its two passes, so shared memory bounds how
//    many lines an SM can hold (~160 lines of 320 FP32 points).  Every byte of it
//    therefore holds line data: tiles are single-stage, the coefficient tables are
//    read through L1 (__ldg, 16-byte vectors), and tile sizes are chosen so that
//    several CTAs share an SM.
//  * FP32: a CTA is one warp on one tile.  FP64, which the FP64 pipe's latency and
//    rate bound, not memory: two warps, one for each half of the tile's lines.
//  * Persistent CTAs walk their tiles (the first is the CTA's index, the next ones
//    come from an atomic counter drawn while the current tile is solved): TMA loads
//    complete on an mbarrier, the tile is solved in place, and TMA stores
//    write it back; the next load is issued as soon as the stores have read shared
//    memory.  Several such CTAs per SM overlap one another's loads, compute and
//    stores.  The last CTA to leave clears the counter for the next launch.
//  * Solvers run in blocks of 8 steps without per-step predicates; the next block's
//    points are requested before the current block's dependent chain, so load
//    latency overlaps the chain.
//  * y/z: a tile is 32 consecutive (x,s) elements of a row at every point of the
//    lines; lane t of a warp solves column t of the [n][32] tile (bank-conflict
//    free).
//  * x: a tile is R whole rows and lane (r, s) solves substrate s of row r; one
//    FP32 substrate alone takes a thread per row and 16-byte accesses.
//  * Every wait is bounded; a timeout sets a device error bit instead of trapping.
#include "field_device.cuh"
#include "pcg_internal.cuh"
#include "sweep_solvers.cuh"

namespace pcg {

namespace {

using namespace solvers;

// ------------------------------------------------------------------ y / z

// The y/z sweep.  A tile is 32 consecutive (x,s) elements at all n points of the
// lines of one outer index; it arrives as nc TMA tensor boxes (32, R) of the field
// described as the 3-D tensor (x*S+s, y, z), all completing on one mbarrier.  The
// CTA solves its lines in place and one thread stores it back with nc box stores; the next
// tile's loads start once the stores have read shared memory.  Loads and compute overlap
// across the CTAs an SM holds.
// Coefficients come from the axis's table (head rows, then per-substrate
// constants), so most points need no coefficient load at all.
//
// SC = 1 (FP64: the step's last sweep, or every sweep of a mesh whose factors are not
// deferred): the stored values are multiplied by the scale factors.
// MC = kMcOut (the step's last sweep with the mass check on): the lanes also sum
// their solved values before the faces are written, into a.mc_tot[S + s].  A
// lane's substrate is the same in every tile when S divides 32 (it then keeps one
// running total and adds it once at the end), else it adds its total per tile.
// BULK (the step's last sweep where bulk_fusable): the bulk update after the faces.
template <typename T, int AXIS, int MC, int SC, bool BULK>
__global__ void __launch_bounds__(sweep_threads<T>(), sizeof(T) == 8 ? 8 : 0) sweep_yz_kernel(SweepArgs a, const __grid_constant__ CUtensorMap tmap)
{
	extern __shared__ __align__(128) unsigned char smem[];
	uint64_t* full = reinterpret_cast<uint64_t*>(smem);
	uint32_t& next = *reinterpret_cast<uint32_t*>(smem + 8);
	T* base = reinterpret_cast<T*>(smem + 128);
	const uint32_t lane = threadIdx.x & 31, half = threadIdx.x >> 5;
	const uint32_t n = a.n, m = line_split<T>(n), S = a.S, R = a.box_rows, nc = a.boxes;
	const uint32_t chunk_elems = R * kLanes;
	if (threadIdx.x == 0)
	{
		dev::mbar_init(full, 1);
		dev::fence_mbar_init();
	}
	__syncthreads();
	dev::pdl_wait();
	bool ok = true;
	MassAcc<T> acc;
	acc.zero();
	const bool per_tile = (kLanes % S) != 0;
	const uint32_t classes = S < kLanes ? S : kLanes;
	// 32-bit tile arithmetic: a launch has fewer than 2^32 tiles
	const uint32_t xblocks = (uint32_t)a.xblocks, tiles = (uint32_t)a.tiles, nouter = tiles / xblocks;
	uint32_t t = blockIdx.x;
	for (uint32_t phase = 0; t < tiles; phase ^= 1)
	{
		const uint32_t x0 = (t % xblocks) * kLanes;
		// y takes its z-planes from the last down: the x sweep that ran just before
		// wrote the highest planes last, and their lines are still in L2
		const uint32_t o = AXIS == 1 ? nouter - 1 - t / xblocks : t / xblocks;
		uint32_t drawn = 0;
		if (threadIdx.x == 0)
		{
			dev::mbar_arrive_expect_tx(full, nc * chunk_elems * (uint32_t)sizeof(T));
			for (uint32_t c = 0; c < nc; c++)
			{
				if (AXIS == 1)
					dev::tma_load_3d(base + c * chunk_elems, &tmap, (int)x0, (int)(c * R), (int)o, full);
				else
					dev::tma_load_3d(base + c * chunk_elems, &tmap, (int)x0, (int)o, (int)(c * R), full);
			}
			drawn = dev::next_ticket(a.ticket);
		}
		// lanes past the row hold zero-filled columns that are never stored
		const uint32_t col = x0 + lane;
		const bool in_row = col < a.row_len;
		const uint32_t s = in_row ? col % S : 0;
		const LineCoef<T> L = line_coef(static_cast<const T*>(a.tab), S, a.head, n, s, half);
		LineScale<T> F {};
		if constexpr (SC != 0)
		{
			T g = T(1);
			if (a.gx)
				g = __ldg(static_cast<const T*>(a.gx) + (in_row ? col : 0));
			if (AXIS == 2 && a.gy)
				g *= __ldg(static_cast<const T*>(a.gy) + (uint64_t)s * a.ny + o);
			F = { g, g * __ldg(static_cast<const T*>(a.sc) + s), true };
		}
		ok = __syncthreads_and(dev::mbar_wait(full, phase));
		if (!ok)
			break;
		solve_tile<T, Strided<T, kLanes, 1>, Strided<T, kLanes, -1>, MC, SC>(
			{ base + lane, 0 }, { base + (n - 1) * kLanes + lane, 0 }, n, half, true, L, F, nullptr, &acc);
		if constexpr ((MC & kMcOut) != 0)
			if (per_tile)
			{
				flush_classes(acc.value(), classes, kLanes, a.mc_tot + S + col % S);
				acc.zero();
			}
		if ((BULK || a.face_mask) && in_row)
		{
			T* mine = half == 0 ? base + lane : base + m * kLanes + lane;
			const uint32_t len = half == 0 ? m : n - m;
			if (a.face_mask)
				fielddev::faces_on_half<T, AXIS>(a, col / S, s, o, mine, len, kLanes, half == 0, half == 0 ? n == m : n > m);
			if constexpr (BULK)
				fielddev::bulk_on_half<T>(a.bulk, (T)a.dt, s, mine, len, kLanes);
		}
		if (threadIdx.x == 0)
			next = drawn;
		dev::fence_proxy_async_smem();
		__syncthreads();
		t = next;
		if (threadIdx.x == 0)
		{
			for (uint32_t c = 0; c < nc; c++)
			{
				if (AXIS == 1)
					dev::tma_store_3d(&tmap, (int)x0, (int)(c * R), (int)o, base + c * chunk_elems);
				else
					dev::tma_store_3d(&tmap, (int)x0, (int)o, (int)(c * R), base + c * chunk_elems);
			}
			dev::bulk_commit();
			dev::bulk_wait_read();
		}
	}
	if constexpr ((MC & kMcOut) != 0)
		if (!per_tile)
			flush_classes(acc.value(), classes, kLanes, a.mc_tot + S + lane % S);
	if (!ok && threadIdx.x == 0)
		atomicOr(a.err, DEV_ERR_WAIT_TIMEOUT);
	if (threadIdx.x == 0)
		dev::bulk_wait_all();
	dev::leave(a.ticket);
}

// ------------------------------------------------------------------ x

// The x sweep: a tile is rows_per_tile whole rows.  Lane (r, s) of a warp
// solves substrate s of row r, points S elements apart in shared
// memory; row pitches are chosen so that the lanes of a warp touch distinct banks.
// ST = S when it is a compile-time constant (accesses with immediate offsets), 0
// for the run-time path, -1 above 32 substrates, where a lane takes several lines
// of the tile's one row in turn.  VEC (one FP32 substrate): a lane per row, 16-byte
// accesses.  MC (the mass check on): the lanes also sum their lines' inputs (kMcIn)
// and, on a 1-D mesh, outputs (kMcOut), added once at the end (per line when S is
// above 32).
template <typename T, int ST, int MC, int SC, bool VEC>
__global__ void __launch_bounds__(sweep_threads<T>(), sizeof(T) == 8 ? 8 : 0) sweep_x_kernel(SweepArgs a)
{
	constexpr bool kWide = ST < 0;
	constexpr int STRIDE = ST > 0 ? ST : 0;
	extern __shared__ __align__(128) unsigned char smem[];
	uint64_t* bar = reinterpret_cast<uint64_t*>(smem);
	uint32_t& next = *reinterpret_cast<uint32_t*>(smem + 8);
	T* tile = reinterpret_cast<T*>(smem + 16);
	const uint32_t lane = threadIdx.x & 31, half = threadIdx.x >> 5;
	const uint32_t R = a.rows_per_tile, S = STRIDE ? (uint32_t)STRIDE : a.S, n = a.n;
	const uint32_t r_local = kWide ? 0 : lane / S, s0 = kWide ? lane : lane % S;
	const uint32_t pitch = (uint32_t)a.smem_pitch;
	const uint32_t row_bytes = (uint32_t)round_up(a.row_len * sizeof(T), 16);
	if (threadIdx.x == 0)
	{
		dev::mbar_init(bar, 1);
		dev::fence_mbar_init();
	}
	__syncthreads();
	dev::pdl_wait();
	LineCoef<T> L = line_coef(static_cast<const T*>(a.tab), S, a.head, n, kWide ? min(s0, S - 1) : s0, half);
	MassAcc<T> ai, ao;
	ai.zero();
	ao.zero();
	const uint32_t tiles = (uint32_t)a.tiles;
	uint32_t t = blockIdx.x;
	bool ok = true;
	for (uint32_t phase = 0; t < tiles; phase ^= 1)
	{
		const uint64_t r0 = (uint64_t)t * R;
		const uint32_t nrows = (uint32_t)(a.rows - r0 < (uint64_t)R ? a.rows - r0 : (uint64_t)R);
		T* g = static_cast<T*>(a.field) + r0 * a.pitch;
		uint32_t drawn = 0;
		if (half == 0)
		{
			if (lane == 0)
				dev::mbar_arrive_expect_tx(bar, nrows * row_bytes);
			__syncwarp();
			if (lane < nrows)
				dev::bulk_g2s(tile + lane * pitch, g + lane * a.pitch, row_bytes, bar);
			if (lane == 0)
				drawn = dev::next_ticket(a.ticket);
		}
		ok = __syncthreads_and(dev::mbar_wait(bar, phase));
		if (!ok)
			break;
		T* row = tile + r_local * pitch;
		if constexpr (VEC)
			solve_tile<T, RowLine, RowLine, MC, 0>({ row }, { row }, n, half, r_local < nrows, L, LineScale<T> {}, &ai, &ao);
		else
			for (uint32_t sb = 0; sb < (kWide ? S : 1u); sb += kLanes)
			{
				const uint32_t s = s0 + sb;
				const bool on = r_local < nrows && (!kWide || s < S);
				if (kWide && sb)
					L = line_coef(static_cast<const T*>(a.tab), S, a.head, n, min(s, S - 1), half);
				LineScale<T> F {};
				if constexpr (SC != 0)
					F = { T(1), __ldg(static_cast<const T*>(a.sc) + min(s, S - 1)), true };
				solve_tile<T, Strided<T, STRIDE, 1>, Strided<T, STRIDE, -1>, MC, SC>(
					{ row + s, S }, { row + (n - 1) * S + s, S }, n, half, on, L, F, &ai, &ao);
				if constexpr (MC != 0 && kWide)
					if (on)
					{
						atomicAdd(a.mc_tot + s, ai.value());
						if ((MC & kMcOut) != 0)
							atomicAdd(a.mc_tot + S + s, ao.value());
						ai.zero();
						ao.zero();
					}
			}
		if (kWide)
			L = line_coef(static_cast<const T*>(a.tab), S, a.head, n, s0, half);
		if (threadIdx.x == 0)
			next = drawn;
		dev::fence_proxy_async_smem();
		__syncthreads();
		t = next;
		if (half == 0)
		{
			if (lane < nrows)
				dev::bulk_s2g(g + lane * a.pitch, tile + lane * pitch, row_bytes);
			dev::bulk_commit();
			dev::bulk_wait_read();
			__syncwarp();
		}
	}
	if constexpr (MC != 0 && !kWide)
	{
		// lanes r * S + s share substrate s
		flush_classes(ai.value(), S, kLanes, a.mc_tot + s0);
		if constexpr ((MC & kMcOut) != 0)
			flush_classes(ao.value(), S, kLanes, a.mc_tot + S + s0);
	}
	if (!ok && threadIdx.x == 0)
		atomicOr(a.err, DEV_ERR_WAIT_TIMEOUT);
	if (half == 0)
		dev::bulk_wait_all();
	dev::leave(a.ticket);
}

// ------------------------------------------------------------------ fused x + y

// The x and y sweeps of a 3-D mesh in one persistent launch, z-slab by z-slab.
// x lines and y lines of a z-plane both lie in that plane, so once the x sweep
// has written the planes of a slab, the y sweep of that slab can start -- while
// the x output is still in L2 (the slabs are a few MB and the y sweep reads
// them a slab or two later).  The y tiles then load from L2 instead of HBM and
// the x output is overwritten in L2 before most of it is ever written back: per
// step the field crosses HBM four times instead of six.  The arithmetic of each
// line is unchanged.
//
// Work items are tickets over a table of segments in ticket order: the x tiles
// of slab k (segment X(k)), and the y tiles of slab k - L after X(k) (lag L).
// A y tile waits until every x tile of its slab has signalled (a per-slab
// counter, released by an x tile after its stores completed and acquired by the
// y tile before its tensor loads).  Tickets are handed out in order and an x
// tile never waits, so every awaited x tile belongs to a running CTA and every
// wait ends; the wait is bounded all the same (DEV_ERR_WAIT_TIMEOUT).  An x tile
// signals once the next tile's loads are in flight (its stores had that long to
// land), and before its CTA waits for any slab.
struct XYArgs
{
	const uint4* segs; // {first ticket, slab | kYSeg, tiles, x tiles of the slab (y segments)}
	uint32_t nseg;
	uint32_t total;    // tickets
	uint32_t planes;   // z-planes per slab
	uint32_t* done;    // [slabs] x tiles signalled, zeroed before the launch
	uint32_t* ticket;
	uint64_t ny, nz;
};
constexpr uint32_t kYSeg = 0x80000000u;

__device__ __forceinline__ uint32_t load_acquire(const uint32_t* p)
{
	uint32_t v;
	asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
	return v;
}

__device__ __forceinline__ void fence_proxy_async_global() { asm volatile("fence.proxy.async.global;" ::: "memory"); }

// Bounded wait for *p >= target (the calling lane only).
__device__ __forceinline__ bool wait_at_least(const uint32_t* p, uint32_t target)
{
	const uint64_t t0 = dev::global_ns();
	while (load_acquire(p) < target)
	{
		if (dev::global_ns() - t0 > dev::kWaitNs)
			return false;
		__nanosleep(100);
	}
	return true;
}

template <typename T, int ST, int MC>
__global__ void __launch_bounds__(sweep_threads<T>())
	sweep_xy_kernel(SweepArgs ax, SweepArgs ay, const __grid_constant__ CUtensorMap tmap, XYArgs f)
{
	extern __shared__ __align__(128) unsigned char smem[];
	uint64_t* bar_x = reinterpret_cast<uint64_t*>(smem);
	uint64_t* bar_y = reinterpret_cast<uint64_t*>(smem + 8);
	uint32_t* s_ticket = reinterpret_cast<uint32_t*>(smem + 16);
	T* buf = reinterpret_cast<T*>(smem + 128);
	const uint32_t tid = threadIdx.x, lane = tid & 31, half = tid >> 5;
	// x: lane (r, s) of either warp solves its half of substrate s of row r of the tile
	const uint32_t S = ST ? (uint32_t)ST : ax.S, nx_pts = ax.n, R = ax.rows_per_tile;
	const uint32_t r_local = lane / S, s = lane % S;
	dev::pdl_wait();
	const uint32_t row_bytes = (uint32_t)round_up(ax.row_len * sizeof(T), 16);
	const LineCoef<T> Lx = line_coef(static_cast<const T*>(ax.tab), S, ax.head, nx_pts, s, half);
	MassAcc<T> ai;
	ai.zero();
	// y
	const uint32_t ny_pts = ay.n, Ry = ay.box_rows, nc = ay.boxes, chunk_elems = Ry * kLanes;
	if (tid == 0)
	{
		dev::mbar_init(bar_x, 1);
		dev::mbar_init(bar_y, 1);
		dev::fence_mbar_init();
	}
	__syncthreads();
	uint32_t phase_x = 0, phase_y = 0;
	int pending = -1; // slab of this CTA's last x tile, not yet signalled
	bool ok = true;
	// signals the pending x tile once its stores have completed
	auto signal = [&]() {
		if (pending < 0)
			return;
		if (half == 0)
		{
			dev::bulk_wait_all();
			fence_proxy_async_global();
		}
		__syncthreads();
		if (tid == 0)
		{
			__threadfence();
			atomicAdd(f.done + pending, 1u);
		}
		pending = -1;
	};
	for (;;)
	{
		if (tid == 0)
			*s_ticket = atomicAdd(f.ticket, 1u);
		__syncthreads();
		const uint32_t t = *s_ticket;
		__syncthreads();
		if (t >= f.total)
			break;
		// the segment holding t (segments are in ticket order)
		uint32_t lo = 0, hi = f.nseg;
		while (hi - lo > 1)
		{
			const uint32_t mid = (lo + hi) / 2;
			if (__ldg(&f.segs[mid].x) <= t)
				lo = mid;
			else
				hi = mid;
		}
		const uint4 seg = __ldg(f.segs + lo);
		const uint32_t u = t - seg.x, slab = seg.y & ~kYSeg;
		if (!(seg.y & kYSeg))
		{
			// x tile u of the slab: rows [r0, r0 + nrows)
			const uint64_t slab_r0 = (uint64_t)slab * f.planes * f.ny;
			const uint64_t slab_r1 = min((uint64_t)(slab + 1) * f.planes, f.nz) * f.ny;
			const uint64_t r0 = slab_r0 + (uint64_t)u * R;
			const uint32_t nrows = (uint32_t)min((uint64_t)R, slab_r1 - r0);
			T* g = static_cast<T*>(ax.field) + r0 * ax.pitch;
			if (half == 0)
			{
				if (lane == 0)
					dev::mbar_arrive_expect_tx(bar_x, nrows * row_bytes);
				__syncwarp();
				if (lane < nrows)
					dev::bulk_g2s(buf + lane * ax.smem_pitch, g + lane * ax.pitch, row_bytes, bar_x);
			}
			signal(); // the previous x tile's stores had this long to complete
			if (!__syncthreads_and(dev::mbar_wait(bar_x, phase_x)))
			{
				ok = false;
				break;
			}
			phase_x ^= 1;
			T* row = buf + r_local * ax.smem_pitch + s;
			solve_tile<T, Strided<T, ST, 1>, Strided<T, ST, -1>, MC, 0>(
				{ row, S }, { row + (nx_pts - 1) * S, S }, nx_pts, half, r_local < nrows, Lx, LineScale<T> {}, &ai);
			dev::fence_proxy_async_smem();
			__syncthreads();
			if (half == 0)
			{
				if (lane < nrows)
					dev::bulk_s2g(g + lane * ax.pitch, buf + lane * ax.smem_pitch, row_bytes);
				dev::bulk_commit();
				dev::bulk_wait_read();
			}
			__syncthreads();
			pending = (int)slab;
		}
		else
		{
			signal(); // never wait on a slab while holding an unsignalled x tile
			bool ready = true;
			if (tid == 0)
			{
				ready = wait_at_least(f.done + slab, seg.w);
				fence_proxy_async_global(); // the tensor loads below follow the acquire
			}
			if (!__syncthreads_and(ready))
			{
				ok = false;
				break;
			}
			// y tile u of the slab: 32 columns at every y of one plane
			const uint32_t xblocks = (uint32_t)ay.xblocks;
			const int x0 = (int)((u % xblocks) * kLanes);
			const int o = (int)((uint64_t)slab * f.planes + u / xblocks);
			if (tid == 0)
			{
				dev::mbar_arrive_expect_tx(bar_y, nc * chunk_elems * (uint32_t)sizeof(T));
				for (uint32_t c = 0; c < nc; c++)
					dev::tma_load_3d(buf + c * chunk_elems, &tmap, x0, (int)(c * Ry), o, bar_y);
			}
			const uint32_t sy = (uint64_t)(x0 + lane) < ay.row_len ? (uint32_t)((x0 + lane) % ay.S) : 0;
			const LineCoef<T> Ly = line_coef(static_cast<const T*>(ay.tab), ay.S, ay.head, ny_pts, sy, half);
			if (!__syncthreads_and(dev::mbar_wait(bar_y, phase_y)))
			{
				ok = false;
				break;
			}
			phase_y ^= 1;
			solve_tile<T, Strided<T, kLanes, 1>, Strided<T, kLanes, -1>, 0, 0>(
				{ buf + lane, 0 }, { buf + (ny_pts - 1) * kLanes + lane, 0 }, ny_pts, half, true, Ly, LineScale<T> {});
			dev::fence_proxy_async_smem();
			__syncthreads();
			if (tid == 0)
			{
				for (uint32_t c = 0; c < nc; c++)
					dev::tma_store_3d(&tmap, x0, (int)(c * Ry), o, buf + c * chunk_elems);
				dev::bulk_commit();
				dev::bulk_wait_read();
			}
			__syncthreads();
		}
	}
	signal();
	if (!ok && tid == 0)
		atomicOr(ax.err, DEV_ERR_WAIT_TIMEOUT);
	if constexpr (MC != 0)
		flush_classes(ai.value(), S, kLanes, ax.mc_tot + s);
	if (half == 0)
		dev::bulk_wait_all();
	dev::leave(f.ticket);
}

struct Plan
{
	uint64_t smem;
	uint64_t rows_per_tile;
	uint64_t pitch; // x: shared-memory row pitch (elements)
};

template <typename T>
Plan plan(const Context* c, int axis)
{
	Plan p {};
	if (axis == 0)
	{
		p.pitch = sweep_x_pitch(c->row_len, c->S, sizeof(T));
		p.rows_per_tile = x_tile_rows(c->row_len, c->S, sizeof(T), x_tile_budget(sizeof(T)));
		p.smem = 16 + p.rows_per_tile * p.pitch * sizeof(T);
		return p;
	}
	uint32_t box_rows, boxes;
	box_geometry(c->n[axis], box_rows, boxes);
	p.smem = 128 + (uint64_t)boxes * box_rows * kLanes * sizeof(T);
	return p;
}

// CTAs of a kernel that an SM holds at once.
int resident_ctas(Context* c, int slot, const void* kernel, int threads, uint64_t smem, uint64_t* per_sm)
{
	Context::Resident& r = c->resident[slot];
	if (r.kernel != kernel || r.smem != smem)
	{
		const int rc = allow_smem(kernel, c->device);
		if (rc)
			return rc;
		int n = 0;
		PCG_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, threads, smem));
		if (n < 1)
			return fail(PCG_ERR_UNSUPPORTED, "sweep tile does not fit in shared memory");
		r = { kernel, smem, n };
	}
	*per_sm = (uint64_t)r.per_sm;
	return PCG_OK;
}

// The grid of a sweep.  Up to two tiles per resident CTA and 16 per SM: a CTA for each
// tile and no counter, whose atomics on one address (two per CTA) take longer than
// the hardware's hand-over of CTAs (steps of sweeps alone, 64^3 x 4: 17.1 -> 15.0 us;
// 240x230x152 x 1, 1.1 waves: 48.3 -> 39.5; but 160x160x320 x 2, 2.1 waves: 69.6 ->
// 73.7, and 40x40x200 x 20, 33 small tiles per SM: 39.0 -> 40.5).  Beyond that
// persistent CTAs draw their tiles, so that a tile's load starts as soon as the last
// one's stores have read shared memory.
int sweep_grid(Context* c, int axis, const void* kernel, int threads, uint64_t smem, SweepArgs& a, uint64_t* grid)
{
	uint64_t per_sm = 0;
	const int rc = resident_ctas(c, axis, kernel, threads, smem, &per_sm);
	if (rc)
		return rc;
	const uint64_t sms = (uint64_t)c->sm_count, resident = per_sm * sms;
	const bool direct = a.tiles <= 2 * resident && a.tiles <= 16 * sms;
	if (direct)
		a.ticket = nullptr;
	*grid = direct ? a.tiles : std::min(resident, a.tiles);
	return PCG_OK;
}

SweepArgs base_args(const Context* c, int axis)
{
	SweepArgs a {};
	a.field = c->field.ptr;
	a.tab = c->coef[axis].ptr;
	a.head = c->coef_head[axis];
	a.S = (uint32_t)c->S;
	a.n = (uint32_t)c->n[axis];
	a.row_len = c->row_len;
	a.pitch = c->pitch;
	a.rows = c->rows;
	a.err = c->h_words;
	a.ticket = static_cast<uint32_t*>(c->tickets.ptr) + 2 * axis;
	a.nx = (uint32_t)c->n[0], a.ny = (uint32_t)c->n[1], a.nz = (uint32_t)c->n[2];
	if (c->wsize == 8)
		a.sc = c->scale_table(axis);
	if (c->wsize == 8 && axis == c->dims - 1 && c->defer_scale)
	{
		// the last sweep applies the earlier axes' factors (their per-point tables
		// follow the S converged ones)
		if (axis > 0)
			a.gx = c->scale_table(0) + c->S;
		if (axis > 1)
			a.gy = c->scale_table(1) + c->S;
	}
	return a;
}

using XKernel = void (*)(SweepArgs);

// The x kernel: S at compile time up to 8, a vector kernel for one FP32 substrate.
template <typename T, int MC>
XKernel x_kernel_by_s(uint64_t S)
{
	switch (S)
	{
	case 1: return sweep_x_kernel<T, 1, MC, 0, sizeof(T) == 4>;
	case 2: return sweep_x_kernel<T, 2, MC, 0, false>;
	case 3: return sweep_x_kernel<T, 3, MC, 0, false>;
	case 4: return sweep_x_kernel<T, 4, MC, 0, false>;
	case 5: return sweep_x_kernel<T, 5, MC, 0, false>;
	case 6: return sweep_x_kernel<T, 6, MC, 0, false>;
	case 7: return sweep_x_kernel<T, 7, MC, 0, false>;
	case 8: return sweep_x_kernel<T, 8, MC, 0, false>;
	default: return S <= kLanes ? sweep_x_kernel<T, 0, MC, 0, false> : sweep_x_kernel<T, -1, MC, 0, false>;
	}
}

// On a 1-D mesh x is also the last sweep: it sums its outputs as well, and an FP64
// sweep that applies its factors itself (1-D, or factors not deferred) takes the
// run-time kernel.
template <typename T>
XKernel x_kernel(const Context* c, bool mass_check)
{
	constexpr int SC = sizeof(T) == 8;
	const bool wide = c->S > kLanes;
	if (c->dims == 1 && mass_check)
		return wide ? sweep_x_kernel<T, -1, kMcIn | kMcOut, SC, false> : sweep_x_kernel<T, 0, kMcIn | kMcOut, SC, false>;
	if (SC && !c->defer_scale && mass_check)
		return wide ? sweep_x_kernel<T, -1, kMcIn, SC, false> : sweep_x_kernel<T, 0, kMcIn, SC, false>;
	if (c->dims == 1 || (SC && !c->defer_scale))
		return wide ? sweep_x_kernel<T, -1, 0, SC, false> : sweep_x_kernel<T, 0, 0, SC, false>;
	return mass_check ? x_kernel_by_s<T, kMcIn>(c->S) : x_kernel_by_s<T, 0>(c->S);
}

template <typename T>
int run_sweep_x(Context* c, bool mass_check)
{
	SweepArgs a = base_args(c, 0);
	const Plan p = plan<T>(c, 0);
	if (p.smem > kMaxSmemBytes)
		return fail(PCG_ERR_UNSUPPORTED, "x rows too long for the shared-memory x sweep");
	a.smem_pitch = p.pitch;
	a.rows_per_tile = (uint32_t)p.rows_per_tile;
	a.tiles = (c->rows + p.rows_per_tile - 1) / p.rows_per_tile;
	if (mass_check)
		a.mc_tot = static_cast<double*>(c->mc_tot.ptr);
	const XKernel kernel = x_kernel<T>(c, mass_check);
	uint64_t grid;
	int rc;
	if ((rc = sweep_grid(c, 0, reinterpret_cast<const void*>(kernel), sweep_threads<T>(), p.smem, a, &grid)))
		return rc;
	cudaEvent_t ev;
	launch_begin(c, K_SWEEP_X, 2.0 * (double)(c->V * c->S) * (double)sizeof(T), &ev);
	PCG_CUDA_TRY(launch_chained(kernel, (unsigned)grid, sweep_threads<T>(), p.smem, c->stream, a));
	launch_end(c, K_SWEEP_X, ev);
	PCG_CUDA_TRY(cudaGetLastError());
	return PCG_OK;
}

// The fused x + y launch (sweep_xy_kernel): slabs of about c->xy_slab_bytes of
// planes, y lagging x by at least c->xy_lag slabs and by at least twice the
// tiles the resident CTAs hold.  The segment table is rebuilt when the slab plan
// changes.
template <typename T>
int run_sweep_xy(Context* c, bool mass_check)
{
	SweepArgs ax = base_args(c, 0);
	const Plan px = plan<T>(c, 0);
	ax.smem_pitch = px.pitch;
	ax.rows_per_tile = (uint32_t)px.rows_per_tile;
	if (mass_check)
		ax.mc_tot = static_cast<double*>(c->mc_tot.ptr);
	SweepArgs ay = base_args(c, 1);
	ay.xblocks = (c->row_len + kLanes - 1) / kLanes;
	ay.box_rows = c->tmap_box_rows[1];
	ay.boxes = c->tmap_boxes[1];
	const Plan py = plan<T>(c, 1);
	const uint64_t R = px.rows_per_tile, ny = c->n[1], nz = c->n[2];
	const uint64_t plane_bytes = ny * c->pitch * sizeof(T);
	const uint64_t P = std::max<uint64_t>(1, std::min<uint64_t>(nz, c->xy_slab_bytes / plane_bytes));
	const uint64_t nslab = (nz + P - 1) / P;
	// the persistent grid (every CTA holds one tile at a time)
	const uint64_t smem = 128 + std::max(px.smem - 16, py.smem - 128);
	if (smem > kMaxSmemBytes)
		return fail(PCG_ERR_UNSUPPORTED, "fused x/y tiles too large for shared memory");
	auto kernel = [&]() -> void (*)(SweepArgs, SweepArgs, const CUtensorMap, XYArgs) {
		const bool mc = mass_check;
		switch (c->S)
		{
		case 3: return mc ? sweep_xy_kernel<T, 3, kMcIn> : sweep_xy_kernel<T, 3, 0>;
		case 4: return mc ? sweep_xy_kernel<T, 4, kMcIn> : sweep_xy_kernel<T, 4, 0>;
		case 5: return mc ? sweep_xy_kernel<T, 5, kMcIn> : sweep_xy_kernel<T, 5, 0>;
		case 6: return mc ? sweep_xy_kernel<T, 6, kMcIn> : sweep_xy_kernel<T, 6, 0>;
		case 7: return mc ? sweep_xy_kernel<T, 7, kMcIn> : sweep_xy_kernel<T, 7, 0>;
		case 8: return mc ? sweep_xy_kernel<T, 8, kMcIn> : sweep_xy_kernel<T, 8, 0>;
		default: return mc ? sweep_xy_kernel<T, 0, kMcIn> : sweep_xy_kernel<T, 0, 0>;
		}
	}();
	uint64_t per_sm = 0;
	int rc;
	if ((rc = resident_ctas(c, 3, reinterpret_cast<const void*>(kernel), sweep_threads<T>(), smem, &per_sm)))
		return rc;
	const uint64_t resident = per_sm * (uint64_t)c->sm_count;
	// the lag must exceed the tiles in flight (about one per resident CTA), else y
	// tiles are handed out while their slab's x tiles are still being solved
	const uint64_t slab_tiles = (P * ny + R - 1) / R + P * ay.xblocks;
	const uint64_t L =
		std::max<uint64_t>(std::max<uint32_t>(1, c->xy_lag), (2 * resident + slab_tiles - 1) / slab_tiles);
	const uint64_t key = P | (L << 20) | (R << 40);
	if (c->xy_key != key || !c->xy_segs.ptr)
	{
		std::vector<uint4> segs;
		uint64_t first = 0;
		std::vector<uint32_t> tx(nslab);
		for (uint64_t k = 0; k < nslab + L; k++)
		{
			if (k < nslab)
			{
				const uint64_t rows_k = (std::min((k + 1) * P, nz) - k * P) * ny;
				tx[k] = (uint32_t)((rows_k + R - 1) / R);
				segs.push_back({ (uint32_t)first, (uint32_t)k, tx[k], 0u });
				first += tx[k];
			}
			if (k >= L)
			{
				const uint64_t j = k - L;
				const uint64_t ty = (std::min((j + 1) * P, nz) - j * P) * ay.xblocks;
				segs.push_back({ (uint32_t)first, (uint32_t)j | kYSeg, (uint32_t)ty, tx[j] });
				first += ty;
			}
		}
		if (first >= 0xffffffffull)
			return fail(PCG_ERR_UNSUPPORTED, "too many tiles for the fused x/y sweep");
		if ((rc = dalloc(c, c->xy_segs, segs.size() * sizeof(uint4))) ||
			(rc = dalloc(c, c->xy_done, nslab * sizeof(uint32_t))))
			return rc;
		PCG_CUDA_TRY(cudaMemcpyAsync(c->xy_segs.ptr, segs.data(), segs.size() * sizeof(uint4), cudaMemcpyHostToDevice,
									 c->stream));
		PCG_CUDA_TRY(stream_wait(c)); // the host table dies at scope exit
		c->xy_key = key;
		c->xy_nseg = (uint32_t)segs.size();
		c->xy_total = (uint32_t)first;
		c->xy_nslab = (uint32_t)nslab;
	}
	XYArgs f {};
	f.segs = static_cast<const uint4*>(c->xy_segs.ptr);
	f.nseg = c->xy_nseg;
	f.total = c->xy_total;
	f.planes = (uint32_t)P;
	f.done = static_cast<uint32_t*>(c->xy_done.ptr);
	f.ticket = static_cast<uint32_t*>(c->tickets.ptr) + 6;
	f.ny = ny;
	f.nz = nz;
	const uint64_t grid = std::min<uint64_t>(resident, c->xy_total);
	PCG_CUDA_TRY(cudaMemsetAsync(f.done, 0, c->xy_nslab * sizeof(uint32_t), c->stream));
	// minimal traffic of the two sweeps: the field read once and written once
	const double bytes = 2.0 * (double)(c->V * c->S) * (double)sizeof(T);
	cudaEvent_t ev;
	launch_begin(c, K_SWEEP_XY, bytes, &ev);
	PCG_CUDA_TRY(launch_chained(kernel, (unsigned)grid, sweep_threads<T>(), smem, c->stream, ax, ay, c->tmap[1], f));
	launch_end(c, K_SWEEP_XY, ev);
	PCG_CUDA_TRY(cudaGetLastError());
	return PCG_OK;
}

// FP64: `scale` when the sweep applies the scale factors (the last one always does).
template <typename T, int AXIS>
auto yz_kernel(bool scale, bool bulk, bool mass_check) -> void (*)(SweepArgs, const CUtensorMap)
{
	constexpr int SC = sizeof(T) == 8;
	if (mass_check)
		return bulk ? sweep_yz_kernel<T, AXIS, kMcOut, SC, true> : sweep_yz_kernel<T, AXIS, kMcOut, SC, false>;
	if (bulk)
		return sweep_yz_kernel<T, AXIS, 0, SC, true>;
	return scale ? sweep_yz_kernel<T, AXIS, 0, SC, false> : sweep_yz_kernel<T, AXIS, 0, 0, false>;
}

template <typename T>
int run_sweep_yz(Context* c, int axis, bool fuse_faces, bool fuse_bulk, bool mass_check)
{
	SweepArgs a = base_args(c, axis);
	if (mass_check)
		a.mc_tot = static_cast<double*>(c->mc_tot.ptr);
	if (fuse_faces)
	{
		const FaceArgs f = make_face_args(c);
		a.face_values = f.values;
		a.face_conds = f.conds;
		a.face_mask = f.face_mask;
	}
	if (fuse_bulk)
	{
		for (int k = 0; k < 3; k++)
			a.bulk[k] = c->bulk[k].ptr;
		a.dt = c->dt;
	}
	a.xblocks = (c->row_len + kLanes - 1) / kLanes;
	a.tiles = a.xblocks * (axis == 1 ? c->n[2] : c->n[1]);
	a.box_rows = c->tmap_box_rows[axis];
	a.boxes = c->tmap_boxes[axis];
	const Plan p = plan<T>(c, axis);
	if (p.smem > kMaxSmemBytes)
		return fail(PCG_ERR_UNSUPPORTED, "lines too long for the shared-memory y/z sweep");
	if (a.box_rows == 0)
		return fail(PCG_ERR_INVALID, "tensor maps of the field were not prepared");
	const int kid = axis == 1 ? K_SWEEP_Y : K_SWEEP_Z;
	const double bytes = 2.0 * (double)(c->V * c->S) * (double)sizeof(T);
	const bool scale = axis == c->dims - 1 || !c->defer_scale;
	auto kernel = axis == 1 ? yz_kernel<T, 1>(scale, fuse_bulk, mass_check)
							: yz_kernel<T, 2>(scale, fuse_bulk, mass_check);
	uint64_t grid;
	int rc;
	if ((rc = sweep_grid(c, axis, reinterpret_cast<const void*>(kernel), sweep_threads<T>(), p.smem, a, &grid)))
		return rc;
	cudaEvent_t ev;
	launch_begin(c, kid, bytes, &ev);
	PCG_CUDA_TRY(launch_chained(kernel, (unsigned)grid, sweep_threads<T>(), p.smem, c->stream, a, c->tmap[axis]));
	launch_end(c, kid, ev);
	PCG_CUDA_TRY(cudaGetLastError());
	return PCG_OK;
}

using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
								   const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
								   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn()
{
	static EncodeTiledFn fn = nullptr;
	if (!fn)
	{
		void* p = nullptr;
		cudaDriverEntryPointQueryResult q {};
		if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
				cudaSuccess &&
			q == cudaDriverEntryPointSuccess)
			fn = reinterpret_cast<EncodeTiledFn>(p);
	}
	return fn;
}

} // namespace

// -------------------------------------------------------------------- host side

// Box geometry of a y/z tile: the fewest TMA boxes of at most 256 points (the box
// limit) that cover a line, each a multiple of the solver block, with the least
// padding.
void box_geometry(uint64_t n, uint32_t& box_rows, uint32_t& boxes)
{
	const uint64_t nc = (n + 255) / 256;
	boxes = (uint32_t)nc;
	box_rows = (uint32_t)round_up((n + nc - 1) / nc, 8);
}

bool x_substrate_mapping(uint64_t S) { return S >= 3 && S <= kLanes; }

// Shared-memory row pitch (elements) of an x tile: whole 16-byte chunks, and rows
// S elements (rounded up to a chunk) apart modulo the 32 banks, so that lane (r, s)
// of a warp reads bank r*S + s (mod 32) for FP32 (two lanes of a bank for S = 2);
// one FP32 substrate alone moves in 16-byte chunks, whose rows lie an odd number of
// chunks apart.  A row that only fits without the padding goes without it.
uint64_t sweep_x_pitch(uint64_t row_len, uint64_t S, size_t wsize)
{
	const uint64_t vn = 16 / wsize;
	const uint64_t mod = 128 / wsize; // elements spanning the 32 banks
	const uint64_t want = round_up(S, vn) % mod;
	uint64_t p = round_up(row_len, vn);
	while (S <= kLanes && p % mod != want)
		p += vn;
	return 16 + p * wsize <= kMaxSmemBytes ? p : round_up(row_len, vn);
}

// Rows of an x tile: one per S lanes of a warp, while the tile stays within
// `budget` bytes.
uint64_t x_tile_rows(uint64_t row_len, uint64_t S, size_t wsize, uint64_t budget)
{
	const uint64_t row_stage = sweep_x_pitch(row_len, S, wsize) * wsize;
	return std::max<uint64_t>(1, std::min<uint64_t>(budget / row_stage, kLanes / S));
}

int encode_field_map(const Context* c, int axis, uint32_t box_rows, CUtensorMap* out, uint32_t box_cols)
{
	EncodeTiledFn enc = encode_fn();
	if (!enc)
		return fail(PCG_ERR_CUDA, "cuTensorMapEncodeTiled is not available from the driver");
	const cuuint64_t dims[3] = { c->row_len, c->n[1], c->n[2] };
	const cuuint64_t strides[2] = { c->pitch * c->wsize, c->n[1] * c->pitch * c->wsize };
	const cuuint32_t estr[3] = { 1, 1, 1 };
	const CUtensorMapDataType dt = c->wsize == 4 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_FLOAT64;
	const cuuint32_t box[3] = { box_cols, axis == 1 ? box_rows : 1u, axis == 2 ? box_rows : 1u };
	CUresult r = enc(out, dt, 3, c->field.ptr, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
					 CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
	if (r != CUDA_SUCCESS)
		return fail(PCG_ERR_CUDA, "cuTensorMapEncodeTiled failed with code " + std::to_string((int)r));
	return PCG_OK;
}

// Encodes the TMA tensor maps of the y and z sweeps for the current field buffer.
int prepare_sweep_maps(Context* c)
{
	for (int axis = 1; axis < c->dims; axis++)
	{
		uint32_t box_rows, boxes;
		box_geometry(c->n[axis], box_rows, boxes);
		const int rc = encode_field_map(c, axis, box_rows, &c->tmap[axis]);
		if (rc)
			return rc;
		c->tmap_box_rows[axis] = box_rows;
		c->tmap_boxes[axis] = boxes;
	}
	return PCG_OK;
}

uint64_t sweep_smem_bytes(const Context* c, int axis)
{
	return c->wsize == 4 ? plan<float>(c, axis).smem : plan<double>(c, axis).smem;
}

int launch_sweep_x(Context* c, bool mass_check)
{
	return c->wsize == 4 ? run_sweep_x<float>(c, mass_check) : run_sweep_x<double>(c, mass_check);
}

bool xy_fusable(const Context* c)
{
	return c->fuse_xy && c->dims == 3 && x_substrate_mapping(c->S) && c->n[2] > 1 && (c->wsize == 4 || c->defer_scale);
}

int launch_sweep_xy(Context* c, bool mass_check)
{
	return c->wsize == 4 ? run_sweep_xy<float>(c, mass_check) : run_sweep_xy<double>(c, mass_check);
}

int launch_sweep_yz(Context* c, int axis, bool fuse_faces, bool fuse_bulk, bool mass_check)
{
	return c->wsize == 4 ? run_sweep_yz<float>(c, axis, fuse_faces, fuse_bulk, mass_check)
						 : run_sweep_yz<double>(c, axis, fuse_faces, fuse_bulk, mass_check);
}

bool faces_fusable(const Context* c) { return c->dims >= 2; }

// Uniform bulk rates in the last sweep's tiles save a pass over the field, but its
// warps are few: with at least three tiles per SM they hide the work (97x131x61 x 5:
// 30.3 -> 26.1 us a step of sweeps and bulk, 64^3 x 4, 512 tiles: 17.4 both, FP64 55 ->
// 51), with fewer they do not (100^3 x 1, 400 tiles: 17.5 -> 19.1; 1000x800 x 3, 94:
// 32 -> 60).  Per-voxel tables measured slower fused at every size (200x200x150 x 4:
// 167 -> 213).  A kernel of its own: a test of the tables in one kernel for both cost
// the sweeps without bulk 2 % (96x80x64 x 20: 68.1 -> 69.5).
bool bulk_fusable(const Context* c)
{
	const uint64_t xblocks = (c->row_len + kLanes - 1) / kLanes, outer = c->dims == 2 ? 1 : c->n[1];
	return c->bulk_mode == PCG_BULK_UNIFORM && faces_fusable(c) && xblocks * outer >= 3 * (uint64_t)c->sm_count;
}

} // namespace pcg
