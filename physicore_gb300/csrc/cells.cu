// cells.cu -- agent secretion/uptake with voxel ballots.
//
// Arithmetic follows openmp_solver/src/cell_solver.cpp:
//   intermediates (51-77)   num = S*T*dt*Vc/Vv, den = (U+S)*dt*Vc/Vv, fac = N*dt/Vv
//   ballot        (79-129)  one winner per voxel collects sum(num), 1+sum(den), sum(fac)
//   result       (131-244)  D' = (D + sum num)/(1 + sum den) + sum fac by the winner;
//                           internalized: fused I += Vv (D - D') when no voxel holds two
//                           agents, otherwise I -= Vv (num - D' den + fac) per agent
//   release      (274-289)  D += I F / Vv, I = 0
//
// GB300 design:
//  * locate: one thread per agent computes its voxel index exactly as
//    cartesian_mesh::voxel_position does (mesh.cpp:37-61; locate in
//    cells_device.cuh: an FP32 estimate decides unless it lies within its error
//    bound of a voxel boundary, where the FP64 division decides), so the
//    agent->voxel maps and the per-voxel counts are bit-exact with the reference.
//  * ballot: a run of lanes in one voxel counts with one atomic, whose returned
//    offset ranks the agents of the voxel; rank 0 wins (the reference's first
//    compare-and-swap wins, cell_solver.cpp:79-101).
//  * group lists the agents of shared voxels and those that write a voxel; reduce
//    adds the terms of the shared ones to a row per voxel with four-value atomics
//    (cell_solver.cpp:102-127); the conflict flag stays on the device, so the step
//    never waits on the host (the Thrust backend copies it back every step,
//    thrust_solver/src/cell_solver.cpp:251-252).
//  * apply (over the agents that write a voxel) and internalize (over the agents
//    of shared voxels) read the flag on the device and take the reference's
//    fused or two-pass branch.  A voxel's substrates are adjacent in the field, so
//    each agent touches one 32-byte sector of densities (S <= 8, FP32).
//  Batches keep the per-warp ballot with atomics (batch.cu).
#include "cells_device.cuh"

namespace pcg {

namespace {

using namespace cellsdev;

// How locate clears the counts for the ballot after it.
enum : int
{
	kClearNone = 0,    // they hold zeros already
	kClearByAgent = 1, // over the voxels that the last ballot recorded: zero everywhere else
	kClearArray = 2,   // every count, four to a thread (threads beyond the agents too)
};

// locate: terms (after new agent data) and voxel of each agent; the step's words
// (conflict flag, list lengths) and the counts start at zero.  Clearing by agent
// writes one scattered word per agent (a 32-byte sector each); the launcher takes it
// when agents are fewer than one per 16 voxels (320x320x256, 200,000 agents: 6 us as a
// kernel of its own, against 16 for the array's 105 MB at the copy bandwidth).
template <typename T>
__global__ void cells_locate_kernel(CellArgs a, int clear, uint64_t V)
{
	dev::pdl_wait();
	const uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
	if (i == 0)
		a.flags[0] = a.flags[1] = a.flags[2] = a.flags[3] = 0;
	if (clear == kClearArray)
	{
		const uint64_t k = 4 * i; // the array starts on a 16-byte boundary
		if (k + 4 <= V)
			*reinterpret_cast<uint4*>(a.counts + k) = make_uint4(0, 0, 0, 0);
		else
			for (uint64_t q = k; q < V; q++)
				a.counts[q] = 0;
	}
	if (i >= a.A)
		return;
	if (clear == kClearByAgent)
	{
		const uint32_t old = a.vox[i];
		if (old < V) // not kNoAgent
			a.counts[old] = 0;
	}
	if (a.terms)
		agent_terms<T>(a, i);
	agent_place(a, i);
}

// ballot: rank of every agent in its voxel; the winner of a voxel that may prove to
// be alone there is marked a winner for now.  Apart from locate, whose FP64
// conversions and loads it would wait for: its atomics (one per agent, 45 us for the
// 4M of the dense workload) are all it does.
template <typename T>
__global__ void cells_ballot_kernel(CellArgs a)
{
	dev::pdl_wait();
	const uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
	const uint32_t v = i < a.A ? a.vox[i] : kNoAgent;
	const uint32_t rank = count_rank(a, v);
	if (i >= a.A)
		return;
	a.role[i] = v == kNoAgent ? kRoleNone : (rank == 0 ? kRoleWinner : kRoleLoser);
	if (v != kNoAgent && rank == 1)
	{
		// this agent's row takes the voxel's sums (FP64 builds: 1 + sum den; FP32 rows
		// hold the bare sum, see fp32_update)
		a.owner[v] = (uint32_t)i;
		T* rn = static_cast<T*>(a.rnum) + i * a.ts;
		T* rd = static_cast<T*>(a.rden) + i * a.ts;
		T* rf = static_cast<T*>(a.rfac) + i * a.ts;
		if (a.joined)
			for (uint64_t k = 0; k < a.ts; k++)
				rn[k] = T(0);
		for (uint64_t s = 0; s < a.S; s++)
		{
			rn[s] = rf[s] = T(0);
			rd[s] = sizeof(T) == 8 ? T(1) : T(0);
		}
	}
}

constexpr unsigned kGroupBlock = 256;

// Consecutive agents of a thread: 8 keep blocks and their atomics few; up to 2^20
// agents 4, for more threads in flight (200,000 agents: 13.5 us with 16, 9.6 with 4).
constexpr uint64_t kGroupWide = 1ull << 20;

// group: final roles (cell_solver.cpp:102-127: every agent but the winner of a shared
// voxel is a conflict); the agents of shared voxels listed in agent order (flags[2])
// and, with a writer list, those that write a voxel (alone or winner; flags[3]).  A
// thread takes Q consecutive agents, of which only the winners need their voxel's
// count.  A block scans its counts and reserves its ranges with one atomic: atomics on
// one address serialise.
template <int Q>
__global__ void __launch_bounds__(kGroupBlock, 6) cells_group_kernel(CellArgs a)
{
	__shared__ uint32_t part[2][kGroupBlock / 32];
	__shared__ uint32_t base[2], total[2];
	__shared__ uint32_t stage[kGroupBlock * Q];
	dev::pdl_wait();
	const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
	const uint64_t i0 = (blockIdx.x * (uint64_t)kGroupBlock + threadIdx.x) * Q;
	const uint32_t n = i0 < a.A ? (uint32_t)min((uint64_t)Q, a.A - i0) : 0u;
	struct alignas(Q) Roles
	{
		uint8_t r[Q];
	} roles {};
	if (n == Q)
		roles = *reinterpret_cast<const Roles*>(a.role + i0);
	else
		for (uint32_t q = 0; q < n; q++)
			roles.r[q] = a.role[i0 + q];
	uint32_t shared = 0, writes = 0; // bit q: agent i0 + q
	uint32_t cnt[Q]; // the winners' voxels, then their counts, all loads of a kind in flight together
#pragma unroll
	for (uint32_t q = 0; q < Q; q++)
		cnt[q] = roles.r[q] == kRoleWinner ? a.vox[i0 + q] : 0u;
#pragma unroll
	for (uint32_t q = 0; q < Q; q++)
		cnt[q] = roles.r[q] == kRoleWinner ? a.counts[cnt[q]] : 0u;
#pragma unroll
	for (uint32_t q = 0; q < Q; q++)
	{
		if (roles.r[q] == kRoleWinner)
		{
			if (cnt[q] == 1)
				roles.r[q] = kRoleAlone;
			else
				a.sums[i0 + q] = a.owner[a.vox[i0 + q]];
			writes |= 1u << q;
		}
		if (roles.r[q] >= kRoleWinner)
			shared |= 1u << q;
	}
	if (n == Q)
		*reinterpret_cast<Roles*>(a.role + i0) = roles;
	else
		for (uint32_t q = 0; q < n; q++)
			a.role[i0 + q] = roles.r[q];
	uint32_t psh = __popc(shared), pwr = a.writers ? __popc(writes) : 0u;
#pragma unroll
	for (uint32_t o = 1; o < 32; o <<= 1)
	{
		const uint32_t t0 = __shfl_up_sync(0xffffffffu, psh, o), t1 = __shfl_up_sync(0xffffffffu, pwr, o);
		if (lane >= o)
			psh += t0, pwr += t1;
	}
	if (lane == 31)
		part[0][warp] = psh, part[1][warp] = pwr;
	__syncthreads();
	if (threadIdx.x == 0)
	{
		uint32_t sum[2] = { 0, 0 };
		for (uint32_t w = 0; w < kGroupBlock / 32; w++)
#pragma unroll
			for (int l = 0; l < 2; l++)
			{
				const uint32_t t = part[l][w];
				part[l][w] = sum[l];
				sum[l] += t;
			}
		// both lists' ranges with one 64-bit atomic on their adjacent words (neither
		// total reaches 2^32, so no carry crosses)
		unsigned long long old = 0ull;
		if (sum[0] | sum[1])
			old = atomicAdd(reinterpret_cast<unsigned long long*>(a.flags + 2),
							((unsigned long long)sum[1] << 32) | (unsigned long long)sum[0]);
		if (sum[0]) // a shared voxel has a loser
			a.flags[0] = 1;
		total[0] = sum[0], total[1] = sum[1];
		base[0] = (uint32_t)old, base[1] = (uint32_t)(old >> 32);
	}
	__syncthreads();
	// the entries, in agent order, through shared memory: a thread's are side by side,
	// so written directly each store of a warp would touch 32 sectors
	for (int list = 0; list < (a.writers ? 2 : 1); list++)
	{
		uint32_t at = list ? part[1][warp] + pwr - __popc(writes) : part[0][warp] + psh - __popc(shared);
		const uint32_t bits = list ? writes : shared;
		uint32_t* to = (list ? a.writers : a.shared) + base[list];
#pragma unroll
		for (uint32_t q = 0; q < Q; q++)
			if ((bits >> q) & 1u)
				stage[at++] = (uint32_t)(i0 + q);
		__syncthreads();
		for (uint32_t k = threadIdx.x; k < total[list]; k += kGroupBlock)
			to[k] = stage[k];
		__syncthreads();
	}
}

// reduce: every agent of a shared voxel adds its terms to its voxel's row.  Four-value atomics run at four times the values per
// second of single ones (4M agents x 12 values on 182,253 voxels: 76 us against 241;
// grouping the agents by voxel and summing each group with warp scans took 128).  A
// warp whose agents all share one voxel (a crowd in one place) sums its terms first
// and adds them once.
template <typename T, int SC>
__global__ void cells_reduce_kernel(CellArgs a)
{
	dev::pdl_wait();
	const uint32_t count = a.flags[a.list_word];
	const uint32_t S = SC ? (uint32_t)SC : (uint32_t)a.S;
	T* rnum = static_cast<T*>(a.rnum);
	T* rden = static_cast<T*>(a.rden);
	T* rfac = static_cast<T*>(a.rfac);
	for (uint64_t j0 = blockIdx.x * (uint64_t)blockDim.x + (threadIdx.x & ~31u); j0 < count;
		 j0 += (uint64_t)gridDim.x * blockDim.x)
	{
		const uint64_t j = j0 + (threadIdx.x & 31);
		uint64_t i = 0;
		uint32_t v = kNoAgent, o = 0;
		if (j < count)
		{
			i = a.shared[j];
			v = a.vox[i];
			o = a.owner[v];
		}
		const T* num = static_cast<const T*>(a.num) + i * a.ts;
		const T* den = static_cast<const T*>(a.den) + i * a.ts;
		const T* fac = static_cast<const T*>(a.fac) + i * a.ts;
		if (__all_sync(0xffffffffu, v == __shfl_sync(0xffffffffu, v, 0)))
		{
			for (uint32_t s = 0; s < S; s++)
			{
				T x[3] = { num[s], den[s], fac[s] };
#pragma unroll
				for (int k = 0; k < 3; k++)
				{
					for (int d = 16; d > 0; d >>= 1)
						x[k] += __shfl_xor_sync(0xffffffffu, x[k], d);
					if ((threadIdx.x & 31) == 0)
						atomicAdd((k == 0 ? rnum : k == 1 ? rden : rfac) + (uint64_t)o * a.ts + s, x[k]);
				}
			}
			continue;
		}
		if (v == kNoAgent)
			continue;
		const uint64_t row = (uint64_t)o * a.ts;
		if (a.joined) // FP32 rows are padded to whole quads
			add_values(rnum + row, num, sizeof(T) == 4 ? (3 * S + 3) / 4 * 4 : 3 * S, true);
		else
		{
			add_values(rnum + row, num, S, a.vec);
			add_values(rden + row, den, S, a.vec);
			add_values(rfac + row, fac, S, a.vec);
		}
	}
}

// FP32: registers capped for 3 blocks of 256 per SM (a latency-bound gather:
// more loads in flight; the FP64 build would spill)
template <typename T>
__global__ void __launch_bounds__(256, sizeof(T) == 4 ? 3 : 1) cells_apply_kernel(CellArgs a)
{
	dev::pdl_wait();
	const uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
	if (i < a.A)
		agent_apply<T>(a, i);
}

// Over the agents that write a voxel (alone or winner; flags[3] of them, listed
// by classify) when they are fewer than half the agents, else over every agent
// (agent_apply returns at once for the others): with many agents per voxel most
// agents only lose their ballot, and a thread per agent would mostly wait on its
// role byte.  Grid-stride, so the grid need not match the device-side count.
// SC: S fixed at compile time (1-8), else 0.
template <typename T, int SC>
__global__ void __launch_bounds__(256, sizeof(T) == 4 ? 3 : 1) cells_apply_writers_kernel(CellArgs a)
{
	dev::pdl_wait();
	const uint32_t count = a.flags[3];
	const bool list = 2ull * count < a.A;
	const uint64_t n = list ? count : a.A;
	for (uint64_t j = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; j < n; j += (uint64_t)gridDim.x * blockDim.x)
		agent_apply<T, SC>(a, list ? a.writers[j] : j);
}

// Over the list of agents in shared voxels (empty when there was no conflict).
template <typename T, int SC>
__global__ void cells_internalize_kernel(CellArgs a)
{
	dev::pdl_wait();
	const uint32_t count = a.flags[a.list_word];
	for (uint64_t j = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; j < count; j += (uint64_t)gridDim.x * blockDim.x)
		agent_internalize<T, SC>(a, a.shared[j]);
}

// Both passes of few agents, one to a thread of one block: the agents of shared voxels
// read the final densities after the barrier.  A launch less (120x120 x 3, 100
// agents: 29.8 -> 28.5 us a step); with two agents to a thread it was slower than the
// two launches (48x40x36 x 2, 1000 agents: 17.1 -> 18.0).
constexpr unsigned kSmallAgents = 256, kSmallBlock = 256;
template <typename T, int SC>
__global__ void __launch_bounds__(kSmallBlock) cells_small_kernel(CellArgs a)
{
	dev::pdl_wait();
	if (threadIdx.x < (uint32_t)a.A)
		agent_apply<T, SC>(a, threadIdx.x);
	__syncthreads();
	if (threadIdx.x < a.flags[a.list_word])
		agent_internalize<T, SC>(a, a.shared[threadIdx.x]);
}

// launch_chained of KERNEL<T, S> for S = 1..8, KERNEL<T, 0> otherwise.
#define PCG_LAUNCH_BY_S(KERNEL, T, S, GRID, BLOCK, STREAM, ARGS)                                                       \
	do                                                                                                                 \
	{                                                                                                                  \
		void (*by_s__[9])(CellArgs) = { KERNEL<T, 0>, KERNEL<T, 1>, KERNEL<T, 2>, KERNEL<T, 3>, KERNEL<T, 4>,          \
										KERNEL<T, 5>, KERNEL<T, 6>, KERNEL<T, 7>, KERNEL<T, 8> };                      \
		PCG_CUDA_TRY(launch_chained(by_s__[(S) <= 8 ? (S) : 0], GRID, BLOCK, 0, STREAM, ARGS));                        \
	} while (0)

// release_internal (cell_solver.cpp:274-289) for one agent
template <typename T>
__global__ void cells_release_kernel(CellArgs a, uint64_t agent)
{
	const uint64_t s = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
	if (s >= a.S)
		return;
	uint32_t idx[3];
	if (!locate(a, agent, idx))
	{
		atomicOr(a.err, DEV_ERR_AGENT_OUTSIDE);
		return;
	}
	T* D = static_cast<T*>(a.field) + ((uint64_t)idx[2] * a.n[1] + idx[1]) * a.pitch + idx[0] * a.S + s;
	const uint64_t k = agent * a.S + s;
	const double I = a.pairs ? pair_value(a.internal[k]) : a.internal[k];
	*D = (T)((double)*D + I * a.frac[k] / a.Vv);
	a.internal[k] = 0.0; // zero bits: a zero pair too
}

} // namespace

namespace cellsdev {

CellArgs make_cell_args(const Context* c)
{
	CellArgs a {};
	a.dims = c->dims;
	a.A = c->A;
	a.S = c->S;
	for (int d = 0; d < 3; d++)
	{
		a.n[d] = c->n[d];
		a.bbmin[d] = (double)c->bbmin[d];
		a.voxel[d] = (double)c->voxel[d];
	}
	a.pitch = c->pitch;
	a.Vv = (double)(c->voxel[0] * c->voxel[1] * c->voxel[2]);
	a.dt = c->dt;
	a.pos = static_cast<const double*>(c->a_pos.ptr);
	a.sec = static_cast<const double*>(c->a_sec.ptr);
	a.sat = static_cast<const double*>(c->a_sat.ptr);
	a.upt = static_cast<const double*>(c->a_upt.ptr);
	a.net = static_cast<const double*>(c->a_net.ptr);
	a.vol = static_cast<const double*>(c->a_vol.ptr);
	a.frac = static_cast<const double*>(c->a_frac.ptr);
	a.active = static_cast<const uint8_t*>(c->a_active.ptr);
	a.internal = static_cast<double*>(c->a_internal.ptr);
	a.vox = static_cast<uint32_t*>(c->a_vox.ptr);
	a.foff = static_cast<uint32_t*>(c->a_foff.ptr);
	// num, den and fac side by side in each agent's row
	const size_t rb = c->S * c->wsize;
	a.ts = c->term_stride;
	a.num = c->a_terms.ptr;
	a.den = static_cast<char*>(c->a_terms.ptr) + rb;
	a.fac = static_cast<char*>(c->a_terms.ptr) + 2 * rb;
	a.rnum = c->a_reduced.ptr;
	a.rden = static_cast<char*>(c->a_reduced.ptr) + rb;
	a.rfac = static_cast<char*>(c->a_reduced.ptr) + 2 * rb;
	a.owner = static_cast<uint32_t*>(c->owner.ptr);
	a.counts = static_cast<uint32_t*>(c->counts.ptr);
	a.role = static_cast<uint8_t*>(c->a_role.ptr);
	a.shared = static_cast<uint32_t*>(c->a_shared.ptr);
	a.flags = static_cast<uint32_t*>(c->flags.ptr);
	a.err = c->h_words;
	a.field = c->field.ptr;
	a.internalized = c->compute_internalized ? 1 : 0;
	a.vec = rows_vectorizable(a, c->wsize);
	a.terms = 1;
	a.pairs = c->wsize == 4 ? 1 : 0; // FP32 contexts store internalized amounts as float pairs
	a.sums = static_cast<uint32_t*>(c->a_sums.ptr);
	a.joined = 1;
	a.writers = static_cast<uint32_t*>(c->a_writers.ptr);
	a.list_word = 2; // (a batch sets 1 for its per-warp ballot)
	set_fast_locate(a);
	return a;
}

} // namespace cellsdev

// The ballot of a single domain (cells_device.cuh) on `stream`; launch bookkeeping
// through `c` when given.  `clear` (kClear*): what is left of the counts of V voxels.
template <typename T>
static int run_ballot(Context* c, const CellArgs& a, int clear, uint64_t V, cudaStream_t stream, int sm_count)
{
	const unsigned block = 256;
	const unsigned grid = (unsigned)((a.A + block - 1) / block);
	const bool wide = a.A > kGroupWide;
	const uint64_t per_block = (uint64_t)kGroupBlock * (wide ? 8 : 4);
	const unsigned ggrid = (unsigned)((a.A + per_block - 1) / per_block);
	// the list of shared-voxel agents is only known on the device: grid-stride
	const unsigned lgrid = std::min<unsigned>(grid, 24 * std::max(sm_count, 1));
	const double S = (double)a.S, A = (double)a.A, w = (double)sizeof(T);
	cudaEvent_t ev = nullptr;
	const uint64_t threads = clear == kClearArray ? std::max<uint64_t>(a.A, (V + 3) / 4) : a.A;
	if (c)
		launch_begin(c, K_CELLS_LOCATE,
					 A * (8.0 * a.dims + 1 + 4 + 4) + (a.terms ? A * (5 * S * 8 + 8 + 3 * S * w) : 0) +
						 (clear == kClearByAgent ? 8 * A : clear == kClearArray ? 4.0 * (double)V : 0.0),
					 &ev);
	PCG_CUDA_TRY(launch_chained(cells_locate_kernel<T>, (unsigned)((threads + block - 1) / block), block, 0, stream, a, clear,
								V));
	if (c)
		launch_end(c, K_CELLS_LOCATE, ev);
	// voxel in, role out, one count updated
	if (c)
		launch_begin(c, K_CELLS_BALLOT, A * (4 + 1 + 8), &ev);
	PCG_CUDA_TRY(launch_chained(cells_ballot_kernel<T>, grid, block, 0, stream, a));
	if (c)
		launch_end(c, K_CELLS_BALLOT, ev);
	// per agent its role in and out; shared-voxel agents and writers: list entry;
	// writers: voxel and count
	if (c)
		launch_begin(c, K_CELLS_GROUP, 2 * A, &ev);
	PCG_CUDA_TRY(launch_chained(wide ? cells_group_kernel<8> : cells_group_kernel<4>, ggrid, kGroupBlock, 0, stream, a));
	if (c && c->timing) // list lengths for the per-agent byte counts
	{
		PCG_CUDA_TRY(
			cudaMemcpyAsync(c->h_words + 2, a.flags + a.list_word, sizeof(uint32_t), cudaMemcpyDeviceToHost, stream));
		PCG_CUDA_TRY(cudaMemcpyAsync(c->h_words + 3, a.flags + 3, sizeof(uint32_t), cudaMemcpyDeviceToHost, stream));
	}
	if (c)
		launch_end(c, K_CELLS_GROUP, ev, 4.0, 12.0);
	// per shared-voxel agent: list entry, voxel, its row's index, role and terms
	if (c)
		launch_begin(c, K_CELLS_REDUCE, 0.0, &ev);
	PCG_LAUNCH_BY_S(cells_reduce_kernel, T, a.S, lgrid, block, stream, a);
	if (c)
		launch_end(c, K_CELLS_REDUCE, ev, 13.0 + 3 * S * w);
	return PCG_OK;
}

template <typename T>
static int run_cells(Context* c, bool recompute)
{
	if (c->A == 0)
		return PCG_OK;
	CellArgs a = make_cell_args(c);
	const unsigned block = 256;
	const unsigned grid = (unsigned)((c->A + block - 1) / block);
	const double S = (double)c->S, A = (double)c->A, w = (double)sizeof(T);
	cudaEvent_t ev;
	// the cached roles and lists must come from this kind of ballot (a batch keeps
	// its own list and counts)
	if (c->ballot_kind != 1)
		recompute = true;
	if (recompute)
	{
		// A captured ballot runs when its graph is replayed, any number of times or never,
		// so it clears the whole array, and a later one relies on nothing it writes.
		cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
		PCG_CUDA_TRY(cudaStreamIsCapturing(c->stream, &capture));
		const bool runs = capture == cudaStreamCaptureStatusNone;
		const int clear = runs && c->counts_follow_vox && c->A * 16 < c->V ? kClearByAgent : kClearArray;
		// the terms (rates, volume in; three rows out) only after new agent data
		a.terms = c->terms_dirty ? 1 : 0;
		const int rc = run_ballot<T>(c, a, clear, c->V, c->stream, c->sm_count);
		if (rc)
			return rc;
		if (runs)
		{
			c->counts_follow_vox = true;
			c->terms_dirty = false;
		}
		c->ballot_kind = 1;
	}
	// per writer: list entry, role, offset, summed (or own) terms, density read and
	// write, internalized amounts read and written
	if (c->compute_internalized && c->A <= kSmallAgents)
	{
		launch_begin(c, K_CELLS_APPLY, 0.0, &ev);
		PCG_LAUNCH_BY_S(cells_small_kernel, T, c->S, 1, kSmallBlock, c->stream, a);
		launch_end(c, K_CELLS_APPLY, ev, 8.0 + 4 * S * w + 16 * S, 9 + 5 * S * w + 16 * S);
		return PCG_OK;
	}
	launch_begin(c, K_CELLS_APPLY, 0.0, &ev);
	const unsigned agrid = std::min<unsigned>(grid, 24 * std::max(c->sm_count, 1));
	PCG_LAUNCH_BY_S(cells_apply_writers_kernel, T, c->S, agrid, block, c->stream, a);
	launch_end(c, K_CELLS_APPLY, ev, 0.0, 9 + 3 * S * w + 2 * S * w + (c->compute_internalized ? 16 * S : 0));
	PCG_CUDA_TRY(cudaGetLastError());
	if (c->compute_internalized)
	{
		// the agents that share a voxel (a few percent at 1e6 agents in 320^3 voxels):
		// list entry, offset, density, own terms, internalized read and write each
		launch_begin(c, K_CELLS_INTERNALIZE, 0.0, &ev);
		const unsigned igrid = std::min<unsigned>(grid, 24 * std::max(c->sm_count, 1));
		PCG_LAUNCH_BY_S(cells_internalize_kernel, T, c->S, igrid, block, c->stream, a);
		launch_end(c, K_CELLS_INTERNALIZE, ev, 8.0 + 4 * S * w + 16 * S);
		PCG_CUDA_TRY(cudaGetLastError());
	}
	return PCG_OK;
}

int launch_cells(Context* c, bool recompute)
{
	return c->wsize == 4 ? run_cells<float>(c, recompute) : run_cells<double>(c, recompute);
}

// The same kernels over caller-owned buffers.
int launch_cells_fp32_buffers(const CellStepBuffers& b, cudaStream_t stream)
{
	if (b.A == 0)
		return PCG_OK;
	CellArgs a {};
	a.dims = b.dims;
	a.A = b.A;
	a.S = b.S;
	for (int d = 0; d < 3; d++)
	{
		a.n[d] = b.n[d];
		a.bbmin[d] = (double)b.bbmin[d];
		a.voxel[d] = (double)b.voxel[d];
	}
	a.pitch = b.pitch;
	a.Vv = (double)(b.voxel[0] * b.voxel[1] * b.voxel[2]);
	a.dt = b.dt;
	a.pos = b.pos;
	a.sec = b.sec;
	a.sat = b.sat;
	a.upt = b.upt;
	a.net = b.net;
	a.vol = b.vol;
	a.frac = nullptr;
	a.active = b.active;
	a.internal = b.internal;
	a.vox = b.vox;
	a.foff = b.foff;
	a.num = b.num;
	a.den = b.den;
	a.fac = b.fac;
	a.rnum = b.rnum;
	a.rden = b.rden;
	a.rfac = b.rfac;
	a.ts = b.S; // separate arrays
	a.owner = b.owner;
	a.counts = b.counts;
	a.role = b.role;
	a.shared = b.shared;
	a.flags = b.flags;
	a.err = b.err;
	a.field = b.field;
	a.internalized = b.internalized;
	a.vec = rows_vectorizable(a, sizeof(float));
	a.terms = 1;
	a.pairs = 0; // the caller's FP64 amounts
	a.sums = b.sums;
	a.joined = 0;
	a.list_word = 2;
	set_fast_locate(a);
	const uint64_t V = b.n[0] * b.n[1] * b.n[2];
	const unsigned block = 256;
	const unsigned grid = (unsigned)((b.A + block - 1) / block);
	int sm_count = 0, dev = 0;
	if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sm_count, cudaDevAttrMultiProcessorCount, dev) !=
												   cudaSuccess)
		sm_count = 0;
	int rc = run_ballot<float>(nullptr, a, kClearArray, V, stream, sm_count);
	if (rc)
		return rc;
	PCG_CUDA_TRY(launch_chained(cells_apply_kernel<float>, grid, block, 0, stream, a));
	if (b.internalized)
		PCG_CUDA_TRY(launch_chained(cells_internalize_kernel<float, 0>, grid, block, 0, stream, a));
	PCG_CUDA_TRY(cudaGetLastError());
	return PCG_OK;
}

template <typename T>
static int run_release(Context* c, uint64_t agent)
{
	CellArgs a = make_cell_args(c);
	cudaEvent_t ev;
	launch_begin(c, K_CELLS_RELEASE, (double)(c->S * 32), &ev);
	cells_release_kernel<T><<<(unsigned)((c->S + 63) / 64), 64, 0, c->stream>>>(a, agent);
	launch_end(c, K_CELLS_RELEASE, ev);
	PCG_CUDA_TRY(cudaGetLastError());
	return PCG_OK;
}

int launch_release(Context* c, uint64_t agent)
{
	return c->wsize == 4 ? run_release<float>(c, agent) : run_release<double>(c, agent);
}

} // namespace pcg
