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
//  * group lists the agents of shared voxels and those that write a voxel; sort puts
//    the shared ones side by side, voxel by voxel, and reduce sums their terms in
//    registers (cell_solver.cpp:102-127); the conflict flag stays on the device, so the step
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
		for (int k = 0; k < 6; k++)
			a.flags[k] = 0;
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
__global__ void cells_ballot_kernel(CellArgs a)
{
	dev::pdl_wait();
	const uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
	const uint32_t v = i < a.A ? a.vox[i] : kNoAgent;
	const uint32_t rank = count_rank(a, v);
	if (i >= a.A)
		return;
	a.role[i] = v == kNoAgent ? kRoleNone : (rank == 0 ? kRoleWinner : kRoleLoser);
	a.rank[i] = rank;
}

constexpr unsigned kGroupBlock = 256;

// Consecutive agents of a thread: 8 keep blocks and their atomics few; up to 2^20
// agents 4, for more threads in flight (200,000 agents: 13.5 us with 16, 9.6 with 4).
constexpr uint64_t kGroupWide = 1ull << 20;

// group: final roles (cell_solver.cpp:102-127: every agent but the winner of a shared
// voxel is a conflict); the agents of shared voxels listed (flags[2]) and, with a
// writer list, those that write a voxel (alone or winner; flags[3]), in agent order
// within a block.  The winner of a shared voxel reserves a run of slots for its agents
// (owner[v] = the first one, flags[4] counts slots) and lists the pieces of the run
// (flags[5]).  A thread takes Q consecutive agents, of which only the winners need
// their voxel's count.  A block scans its counts and reserves its ranges with two
// atomics: atomics on one address serialise.
template <int Q>
__global__ void __launch_bounds__(kGroupBlock, 5) cells_group_kernel(CellArgs a)
{
	constexpr int kLists = 4; // shared agents, writers, slots, pieces
	__shared__ uint32_t part[kLists][kGroupBlock / 32];
	__shared__ uint32_t base[kLists], total[2];
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
	uint32_t own[kLists] = {};
#pragma unroll
	for (uint32_t q = 0; q < Q; q++)
	{
		if (roles.r[q] == kRoleWinner)
		{
			writes |= 1u << q;
			if (cnt[q] == 1)
			{
				roles.r[q] = kRoleAlone;
				cnt[q] = 0;
			}
		}
		if (roles.r[q] >= kRoleWinner)
			shared |= 1u << q;
		own[2] += cnt[q]; // of shared voxels only
		own[3] += pieces_of(cnt[q]);
	}
	if (n == Q)
		*reinterpret_cast<Roles*>(a.role + i0) = roles;
	else
		for (uint32_t q = 0; q < n; q++)
			a.role[i0 + q] = roles.r[q];
	own[0] = __popc(shared);
	own[1] = a.writers ? __popc(writes) : 0u;
	uint32_t at[kLists];
#pragma unroll
	for (int l = 0; l < kLists; l++)
	{
		at[l] = own[l];
#pragma unroll
		for (uint32_t o = 1; o < 32; o <<= 1)
		{
			const uint32_t t = __shfl_up_sync(0xffffffffu, at[l], o);
			if (lane >= o)
				at[l] += t;
		}
		if (lane == 31)
			part[l][warp] = at[l];
		at[l] -= own[l];
	}
	__syncthreads();
	if (threadIdx.x == 0)
	{
		uint32_t sum[kLists] = {};
		for (uint32_t w = 0; w < kGroupBlock / 32; w++)
#pragma unroll
			for (int l = 0; l < kLists; l++)
			{
				const uint32_t t = part[l][w];
				part[l][w] = sum[l];
				sum[l] += t;
			}
		// two ranges with each 64-bit atomic on adjacent words (no total reaches 2^32,
		// so no carry crosses)
#pragma unroll
		for (int l = 0; l < kLists; l += 2)
		{
			unsigned long long old = 0ull;
			if (sum[l] | sum[l + 1])
				old = atomicAdd(reinterpret_cast<unsigned long long*>(a.flags + 2 + l),
								((unsigned long long)sum[l + 1] << 32) | (unsigned long long)sum[l]);
			base[l] = (uint32_t)old, base[l + 1] = (uint32_t)(old >> 32);
		}
		if (sum[0]) // a shared voxel has a loser
			a.flags[0] = 1;
		total[0] = sum[0], total[1] = sum[1];
	}
	__syncthreads();
	// the entries, in agent order, through shared memory: a thread's are side by side,
	// so written directly each store of a warp would touch 32 sectors
	for (int list = 0; list < (a.writers ? 2 : 1); list++)
	{
		uint32_t k = part[list][warp] + (list ? at[1] : at[0]);
		const uint32_t bits = list ? writes : shared;
		uint32_t* to = (list ? a.writers : a.shared) + base[list];
#pragma unroll
		for (uint32_t q = 0; q < Q; q++)
			if ((bits >> q) & 1u)
				stage[k++] = (uint32_t)(i0 + q);
		__syncthreads();
		for (uint32_t k = threadIdx.x; k < total[list]; k += kGroupBlock)
			to[k] = stage[k];
		__syncthreads();
	}
	uint32_t slot = base[2] + part[2][warp] + at[2], piece = base[3] + part[3][warp] + at[3];
#pragma unroll
	for (uint32_t q = 0; q < Q; q++)
	{
		const uint32_t np = pieces_of(cnt[q]);
		if (np)
		{
			a.owner[a.vox[i0 + q]] = slot;
			if (np <= 4)
				for (uint32_t c = 0; c < np; c++)
					a.pieces[piece + c] = make_piece(slot, cnt[q], c);
		}
		// a crowd's pieces by the whole warp
		for (uint32_t crowds = __ballot_sync(0xffffffffu, np > 4); crowds; crowds &= crowds - 1)
		{
			const int l = __ffs(crowds) - 1;
			const uint32_t s0 = __shfl_sync(0xffffffffu, slot, l), k0 = __shfl_sync(0xffffffffu, cnt[q], l),
						   p0 = __shfl_sync(0xffffffffu, piece, l);
			for (uint32_t c = lane; c < pieces_of(k0); c += 32)
				a.pieces[p0 + c] = make_piece(s0, k0, c);
		}
		slot += cnt[q];
		piece += np;
	}
}

// sort: every agent of a shared voxel takes its slot of the voxel's run.  The rows of
// voxels of several pieces, which add to them, start at zero.  Four consecutive agents
// a thread, found by their roles: over the list, with an agent a turn, the chain from
// entry to voxel to slot took 46 us for the 4M agents of the dense workload, 42
// this way: two random words of L2 per agent.
template <typename T>
__global__ void cells_sort_kernel(CellArgs a)
{
	dev::pdl_wait();
	const uint64_t i0 = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) * 4;
	if (i0 >= a.A)
		return;
	const uint32_t n = (uint32_t)min((uint64_t)4, a.A - i0);
	Values<uint8_t, 4> role {};
	Values<uint32_t, 4> vox {}, rank {};
	if (n == 4)
	{
		role = *reinterpret_cast<const Values<uint8_t, 4>*>(a.role + i0);
		if (max(max(role.t[0], role.t[1]), max(role.t[2], role.t[3])) < kRoleWinner)
			return;
		vox = *reinterpret_cast<const Values<uint32_t, 4>*>(a.vox + i0);
		rank = *reinterpret_cast<const Values<uint32_t, 4>*>(a.rank + i0);
	}
	else
		for (uint32_t q = 0; q < n; q++)
			role.t[q] = a.role[i0 + q], vox.t[q] = a.vox[i0 + q], rank.t[q] = a.rank[i0 + q];
	uint32_t first[4];
#pragma unroll
	for (int q = 0; q < 4; q++)
		first[q] = role.t[q] >= kRoleWinner ? a.owner[vox.t[q]] : 0u;
#pragma unroll
	for (int q = 0; q < 4; q++)
	{
		if (role.t[q] < kRoleWinner)
			continue;
		a.sorted[first[q] + rank.t[q]] = (uint32_t)(i0 + q);
		if (rank.t[q] != 0 || a.counts[vox.t[q]] <= kPiece)
			continue;
		T* rows[3] = { static_cast<T*>(a.rnum), static_cast<T*>(a.rden), static_cast<T*>(a.rfac) };
		for (int k = 0; k < (a.joined ? 1 : 3); k++)
			for (uint64_t s = 0; s < (a.joined ? a.ts : a.S); s++)
				rows[k][(i0 + q) * a.ts + s] = T(0);
	}
}

// N values side by side of the rows of `count` agents of `list` (1 to 8), summed in pairs.
template <typename T, int N>
__device__ __forceinline__ void sum_rows(const T* rows, uint64_t ts, const uint32_t* list, uint32_t count, T (&s)[N])
{
	uint32_t i[8];
	Values<T, N> x[8];
#pragma unroll
	for (uint32_t k = 0; k < 8; k++)
		i[k] = k < count ? list[k] : 0u;
#pragma unroll
	for (uint32_t k = 0; k < 8; k++)
		if (k < count)
			x[k] = *reinterpret_cast<const Values<T, N>*>(rows + i[k] * ts);
		else
			x[k] = Values<T, N> {};
#pragma unroll
	for (int n = 0; n < N; n++)
	{
		s[n] = x[0].t[n] + x[1].t[n];
		if (count > 2)
			s[n] += x[2].t[n] + x[3].t[n];
		if (count > 4)
		{
			T u = x[4].t[n] + x[5].t[n];
			if (count > 6)
				u += x[6].t[n] + x[7].t[n];
			s[n] += u;
		}
	}
}

// Values [e, e + N) of a piece's rows: summed in pairs (at most five roundings for 32
// agents) and stored to the winner's row, or added to it where the voxel has several
// pieces.
template <typename T, int N>
__device__ __forceinline__ void reduce_piece(const CellArgs& a, uint2 piece, uint32_t e, uint32_t S)
{
	const uint32_t len = piece_len(piece), c = piece_number(piece);
	const uint32_t* list = a.sorted + piece.x + c * kPiece;
	const uint32_t arr = N == 1 ? e / S : 0, s0 = N == 1 ? e % S : e; // N == 1: three arrays
	const T* rows = static_cast<const T*>(arr == 0 ? a.num : arr == 1 ? a.den : a.fac) + s0;
	T* to = static_cast<T*>(arr == 0 ? a.rnum : arr == 1 ? a.rden : a.rfac) + s0 + a.sorted[piece.x] * a.ts;
	Values<T, N> sum;
	T u[N], w[N];
	sum_rows<T, N>(rows, a.ts, list, min(len, 8u), sum.t);
	if (len > 8)
	{
		sum_rows<T, N>(rows, a.ts, list + 8, min(len - 8, 8u), u);
#pragma unroll
		for (int n = 0; n < N; n++)
			sum.t[n] += u[n];
	}
	if (len > 16)
	{
		sum_rows<T, N>(rows, a.ts, list + 16, min(len - 16, 8u), u);
		if (len > 24)
		{
			sum_rows<T, N>(rows, a.ts, list + 24, len - 24, w);
#pragma unroll
			for (int n = 0; n < N; n++)
				u[n] += w[n];
		}
#pragma unroll
		for (int n = 0; n < N; n++)
			sum.t[n] += u[n];
	}
	if (sizeof(T) == 8 && c == 0) // FP64 rows hold 1 + sum den, FP32 rows the bare sum (fp32_update)
#pragma unroll
		for (int n = 0; n < N; n++)
			if (e + n >= S && e + n < 2 * S)
				sum.t[n] += T(1);
	if (piece_alone(piece))
		*reinterpret_cast<Values<T, N>*>(to) = sum;
	else
		add_values(to, sum.t);
}

// reduce: the sums of every shared voxel (cell_solver.cpp:102-127), a thread for 16
// bytes of the rows of a piece (a value of one of the three arrays where they are
// apart).  Bound by the gather of rows in random order (4M agents, 182,253 voxels, S = 4:
// 90 us, 6 blocks per SM with fewer registers 114).  One atomic per agent and quad takes
// the same 90 us and no sort, but rounds the sum of k agents k times (1.3e-5 off at
// 1,000 equal agents in FP32) and serialises on crowds (a ballot of 1M agents in 4 voxels, S = 4:
// 1,231 us against 198; FP64 3,423 against 291).
template <typename T, int SC>
__global__ void __launch_bounds__(256) cells_reduce_kernel(CellArgs a)
{
	dev::pdl_wait();
	constexpr int N = 16 / sizeof(T);
	const uint32_t S = SC ? (uint32_t)SC : (uint32_t)a.S;
	const uint32_t np = a.flags[5], parts = a.joined ? (3 * S + N - 1) / N : 3 * S;
	const uint64_t items = (uint64_t)np * parts, stride = (uint64_t)gridDim.x * blockDim.x;
	for (uint64_t w = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; w < items; w += stride)
	{
		const uint2 piece = a.pieces[w / parts];
		const uint32_t q = (uint32_t)(w % parts);
		if (a.joined)
			reduce_piece<T, N>(a, piece, q * N, S);
		else
			reduce_piece<T, 1>(a, piece, q, S);
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
// by group) when they are fewer than half the agents, else over every agent
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
	a.rank = static_cast<uint32_t*>(c->a_order.ptr);
	a.sorted = a.rank + round_up(c->A, 4); // each on a 16-byte boundary
	a.pieces = reinterpret_cast<uint2*>(a.sorted + round_up(c->A, 4));
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
	// the number of pieces, at most A / 2 (a shared voxel holds two agents or more), is
	// only known on the device: grid-stride
	const uint64_t parts = a.joined ? a.ts * sizeof(T) / 16 : 3 * a.S;
	const unsigned rgrid =
		(unsigned)std::min<uint64_t>((a.A / 2 * parts + block) / block, 24 * (uint64_t)std::max(sm_count, 1));
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
	// voxel in, role and rank out, one count updated
	if (c)
		launch_begin(c, K_CELLS_BALLOT, A * (4 + 1 + 4 + 8), &ev);
	PCG_CUDA_TRY(launch_chained(cells_ballot_kernel, grid, block, 0, stream, a));
	if (c)
		launch_end(c, K_CELLS_BALLOT, ev);
	// per agent its role in and out; shared-voxel agents and writers: list entry;
	// writers: voxel and count (and, in shared voxels, first slot and pieces)
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
	// per agent its role; per shared-voxel agent: voxel, rank, its voxel's first slot; its slot
	if (c)
		launch_begin(c, K_CELLS_SORT, A, &ev);
	PCG_CUDA_TRY(launch_chained(cells_sort_kernel<T>, (unsigned)((a.A + 4 * block - 1) / (4 * block)), block, 0, stream, a));
	if (c)
		launch_end(c, K_CELLS_SORT, ev, 16.0);
	// per shared-voxel agent: slot and terms
	if (c)
		launch_begin(c, K_CELLS_REDUCE, 0.0, &ev);
	PCG_LAUNCH_BY_S(cells_reduce_kernel, T, a.S, rgrid, block, stream, a);
	if (c)
		launch_end(c, K_CELLS_REDUCE, ev, 4.0 + 3 * S * w);
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
	a.rank = b.rank;
	a.sorted = b.sorted;
	a.pieces = b.pieces;
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
