/*
 * resident.cu -- the whole solver stage of one step in one launch, its constraint rows
 * held on chip from preparation to impulse storage.
 *
 * Why: a step of the reference solver (src/solver.c:559-731) is a chain of about 110
 * dependent sweeps (per substep: integrate, warm start per colour, solve per colour,
 * integrate positions, relax per colour; then restitution per colour).  A sweep touches
 * well under a megabyte, so a launch per sweep waits on launches: 4.1 us a launch
 * whether a set has 900 or 60000 contacts.  One resident kernel with a barrier between
 * sweeps pays the barrier and the row's own dependent chain instead.
 *
 * Spaces (template parameter CL):
 *   CL == 1   one CTA: rows and body states in its shared memory, __syncthreads between
 *             sweeps.
 *   CL > 1    a thread-block cluster of CL CTAs: rows in the shared memory of the CTA
 *             that solves them, body b in CTA b / block with copies in the CTAs whose
 *             rows touch it, between which updates are passed (b2g_push.h); where the copies
 *             do not fit, reached through distributed shared memory, with hardware
 *             cluster barriers.
 *   CL == 0   a cooperative grid of up to one CTA per SM: rows in shared memory while
 *             they fit (in the world's row arrays otherwise), body states in global
 *             memory read and written at L2; a counter barrier in global memory, every
 *             wait of which is bounded.
 *
 * Row i of colour c belongs to CTA k with first(k) <= i < first(k + 1), first(k) =
 * n * k / CTAs: no two rows of a colour share a non-static body
 * (src/constraint_graph.c:84-131), so any split gives the same bits.  The overflow
 * colour's rows all belong to CTA 0, whose thread 0 solves them in order, on local
 * copies of their bodies when the bodies live elsewhere.
 *
 * Arithmetic is b2g_solve.h's, shared with the per-phase kernels, so every path gives
 * the same bits.
 *
 * What bounds it: the chain of sweeps.  Per sweep 0.33 us in one CTA (0.5 us at 200 rows
 * a colour), 0.6 us in a cluster with body copies and 0.75 to 1 us without, 2 us in a
 * grid (an L2 round trip to arrive and one to see it).  b2SolveContacts, one kernel per
 * phase before and one resident kernel now, four substeps: 900 contacts 420 -> 52 us (a
 * cluster without copies takes 82), 15000 420 -> 102 without copies (a grid takes 199),
 * 60000 424 -> 206; with 17 overflow rows at 15000 contacts 799 -> 185, with body copies
 * 162.
 */
#include "b2g_push.h"
#include "b2g_resident.h"

#include <string.h>

/* The solver stage on caller buffers: one CTA or one cluster.  Body indices are whatever
 * the caller numbered, so the CTAs first find the largest one; when the states up to it
 * do not fit in the cluster's shared memory, they stay in global memory.  Only listed
 * and touched bodies are written back. */
template <int CL, int T>
__global__ void __launch_bounds__( T, 1 ) k_solve_cluster( const __grid_constant__ b2gDevWorld W, const __grid_constant__ ResidentPlan P,
														   const __grid_constant__ b2gStepConst sc )
{
	extern __shared__ float4 smem[];
	__shared__ ResShare share[B2G_COLORS];
	__shared__ int s_rows, s_awake, s_top, s_ovSlots;
	__shared__ PushShared push;
	cg::cluster_group cl = cg::this_cluster();
	const int rank = CL == 1 ? 0 : (int)cl.block_rank();
	const int tid = threadIdx.x;
	const int* cs = P.colorStart;
	SmemRows m = res_carve_rows( smem, P.rowCap );
	ResBodies rb = res_carve_bodies( smem + 9 * P.rowCap, P.bodyCap );
	float4* gst = (float4*)W.state;

	if ( tid < B2G_OVERFLOW )
	{
		int n = cs[tid + 1] - cs[tid];
		int f = res_first( n, rank, CL );
		share[tid].first = cs[tid] + f;
		share[tid].count = res_first( n, rank + 1, CL ) - f;
	}
	if ( tid == 0 )
	{
		s_awake = 0;
		s_top = -1;
		s_ovSlots = 0;
	}
	for ( int s = tid; s < P.bodyCap; s += T )
		rb.flags[s] = 0;
	__syncthreads();
	if ( tid == 0 )
	{
		int base = 0;
		for ( int c = 0; c < B2G_OVERFLOW; ++c )
		{
			share[c].base = base;
			base += share[c].count;
		}
		int ov = rank == 0 ? cs[B2G_COLORS] - cs[B2G_OVERFLOW] : 0;
		share[B2G_OVERFLOW].first = cs[B2G_OVERFLOW];
		share[B2G_OVERFLOW].count = ov;
		share[B2G_OVERFLOW].base = base;
		s_rows = base + ov;
	}
	__syncthreads();
	const int rows = s_rows, colourRows = share[B2G_OVERFLOW].base;

	/* rows, and the largest body index of this CTA's rows and share of the list */
	const int af = res_first( P.awakeCount, rank, CL ), al = res_first( P.awakeCount, rank + 1, CL );
	int top = -1;
	prepare_rows( W, m, rows, nullptr, nullptr, ResSource{ share, 0 }, tid, T, sc );
	for ( int k = tid; k < rows; k += T )
		top = max( top, max( m.idx[k].x, m.idx[k].y ) );
	for ( int i = af + tid; i < al; i += T )
		top = max( top, W.awake[i] );
	top = __reduce_max_sync( 0xffffffffu, top );
	if ( ( tid & 31 ) == 0 )
		atomicMax( &s_top, top );
	if constexpr ( CL > 1 )
	{
		cl.sync();
		/* every CTA reads every CTA's maximum; nothing changes them any more */
		for ( int r = 0; r < CL; ++r )
			top = max( top, *cl.map_shared_rank( &s_top, r ) );
		top = __reduce_max_sync( 0xffffffffu, top );
	}
	else
	{
		__syncthreads();
		top = s_top;
	}

	ResBarrier<CL> bar{ nullptr, CL, 0 };
	const ResJoints J{};
	ResOverflow ov = res_carve_overflow( smem + P.ovOffset, P.ovOffset ? cs[B2G_COLORS] - cs[B2G_OVERFLOW] : 0, 0 );
	auto index_overflow = [&]() {
		if ( CL > 1 && rank == 0 && P.ovOffset )
		{
			res_index_overflow<T, false>( ov, m, J, share[B2G_OVERFLOW], 0, cs[B2G_COLORS] - cs[B2G_OVERFLOW], &s_ovSlots );
			__syncthreads();
		}
	};
	const int ids = top + 1;
	const int block = ids > 0 ? ( ids + CL - 1 ) / CL : 1;
	/* owners by a multiply-high with ceil(2^32 / block): exact for ids below 2^16 */
	if ( block <= P.bodyCap && ids < 65536 )
	{
		const unsigned inv = block > 1 ? (unsigned)( ( ( 1ull << 32 ) + (unsigned)block - 1 ) / (unsigned)block ) : 0u;
		const int owned = min( block, ids - rank * block );
		auto place = [&]( int b, int& r, int& s ) {
			r = CL == 1 ? 0 : ( block == 1 ? b : (int)__umulhi( (unsigned)b, inv ) );
			s = b - r * block;
		};
		auto there = [&]( int* p, int r ) { return CL == 1 ? p : cl.map_shared_rank( p, r ); };
		auto mark_and_load = [&]() {
			for ( int k = tid; k < rows; k += T )
			{
				int4 ix = m.idx[k];
				int r, s;
				if ( ix.x >= 0 )
				{
					place( ix.x, r, s );
					atomicOr( there( rb.flags + s, r ), RES_TOUCHED );
				}
				if ( ix.y >= 0 )
				{
					place( ix.y, r, s );
					atomicOr( there( rb.flags + s, r ), RES_TOUCHED );
				}
			}
			/* the listed bodies to their owners' lists, each once */
			for ( int i = af + tid; i < al; i += T )
			{
				int b = W.awake[i];
				if ( b < 0 )
					continue;
				int r, s;
				place( b, r, s );
				if ( atomicOr( there( rb.flags + s, r ), RES_AWAKE ) & RES_AWAKE )
					continue;
				*there( rb.awake + atomicAdd( there( &s_awake, r ), 1 ), r ) = s;
			}
			for ( int s = tid; s < owned; s += T )
			{
				int b = rank * block + s;
				rb.st0[s] = gst[2 * b];
				rb.st1[s] = gst[2 * b + 1];
			}
		};
		auto clear = [&]() {
			for ( int s = tid; s < block; s += T )
				rb.flags[s] = 0;
			if ( tid == 0 )
				s_awake = 0;
		};
		/* a cluster whose CTAs can hold copies of the bodies that their rows touch; states
		 * in their owners' CTAs only where they cannot */
		bool pushes = false, lost = false;
		PushBodies PB;
		int* ovList = nullptr;
		if constexpr ( CL > 1 )
		{
			const int space = P.pushBytes - PUSH_OWNED_BYTES * block - 8 * ( cs[B2G_COLORS] - cs[B2G_OVERFLOW] );
			const int cap = min( space / PUSH_COPY_BYTES, 65535 );
			if ( space > 0 && cap > block )
			{
				push_carve( smem + 9 * P.rowCap, cap, block, rank, PB, rb );
				push_init( PB, push, P, block );
				ovList = rb.awake + block;
				clear();
				cl.sync();
				mark_and_load();
				pushes = push_exchange<false>( cl, PB, push, cap, block, inv, rows, 0, share, m, J, ovList, rb,
											   s_awake, [&]( int s ) { return ( rb.flags[s] & RES_AWAKE ) != 0; } );
				if ( pushes == false )
				{
					rb = res_carve_bodies( smem + 9 * P.rowCap, P.bodyCap );
					clear();
					cl.sync();
				}
			}
		}
		if ( pushes == false )
		{
			index_overflow();
			mark_and_load();
		}
		bar.sync();
		const int awake = s_awake;
		for ( int j = tid; j < awake; j += T )
			res_terms( W, rb, rb.awake[j], rank * block + rb.awake[j], sc );
		if constexpr ( CL == 1 )
		{
			LocalBodies LB;
			LB.st0 = rb.st0;
			LB.st1 = rb.st1;
			/* a thread's terms are its own: no barrier before the first integration */
			res_run<CL, T, true, false>( P, share, m, J, LB, rb, gst, nullptr, awake, bar, rank, sc, ov, s_ovSlots );
		}
		else if ( pushes )
		{
			push_run<T, false>( P, share, m, J, PB, push, rb, awake, push.copies - block, ovList, sc );
			lost = push_end( cl, push );
		}
		else
		{
			const DsmemBodies D{ { cl, rb.st0, rb.st1, block, rank, inv } };
			res_run<CL, T, true, false>( P, share, m, J, D, rb, gst, nullptr, awake, bar, rank, sc, ov, s_ovSlots );
		}
		for ( int s = tid; s < owned; s += T )
		{
			int b = rank * block + s;
			int f = rb.flags[s];
			/* a cluster of which a CTA gave up on another has no result */
			if ( lost )
				rb.st0[s].x = rb.st0[s].y = rb.st0[s].z = __int_as_float( 0x7fffffff );
			if ( f )
				gst[2 * b] = rb.st0[s];
			if ( f & RES_AWAKE )
				gst[2 * b + 1] = rb.st1[s];
		}
	}
	else
	{
		index_overflow();
		/* states at L2; the terms of this CTA's share of the list, which fit (res_body_cap) */
		L2Bodies G{ gst };
		const int n = al - af;
		for ( int j = tid; j < n; j += T )
			res_terms( W, rb, j, W.awake[af + j], sc );
		bar.sync();
		res_run<CL, T, false, false>( P, share, m, J, G, rb, gst, W.awake + af, n, bar, rank, sc, ov, s_ovSlots );
	}
	store_impulses( W, m, rows, colourRows, tid, T );
}

/* CTAs of a grid that ended before this one. */
__device__ __forceinline__ int grid_ended( int* ctl )
{
	int n;
	asm volatile( "atom.acq_rel.gpu.global.add.s32 %0, [%1], 1;" : "=r"( n ) : "l"( ctl + 1 ) : "memory" );
	return n;
}

/* A grid of which a CTA gave up on another has no result: NaN velocities of the listed bodies
 * and of those with contacts, by one thread, as it is hardly ever called. */
__device__ __noinline__ void mark_lost( const b2gDevWorld& W, int listed, int contacts )
{
	float* st = (float*)W.state;
	for ( int i = 0; i < listed + 2 * contacts; ++i )
	{
		const int b = i < listed ? W.awake[i] : W.cBodies[i - listed];
		for ( int k = 0; k < 3 && b >= 0; ++k )
			st[8 * (size_t)b + k] = __int_as_float( 0x7fffffff );
	}
}

/* The solver stage over a cooperative grid: body states in global memory, rows in shared
 * memory (ONCHIP) or in the row arrays, where row k of the colour-major order is entry k.
 * ctl: the barrier's arrival count, the count of finished CTAs and the give-up flag, all
 * zero at the launch. */
template <int T, bool ONCHIP>
__global__ void __launch_bounds__( T, 1 ) k_solve_grid( const __grid_constant__ b2gDevWorld W, const __grid_constant__ ResidentPlan P,
														const __grid_constant__ b2gStepConst sc, int* ctl )
{
	extern __shared__ float4 smem[];
	__shared__ ResShare share[B2G_COLORS];
	__shared__ int s_ovSlots;
	const int rank = blockIdx.x, ctas = gridDim.x, tid = threadIdx.x;
	const int* cs = P.colorStart;
	const int ovRows = cs[B2G_COLORS] - cs[B2G_OVERFLOW];
	if ( tid == 0 )
	{
		int base = 0;
		for ( int c = 0; c < B2G_COLORS; ++c )
		{
			int n = cs[c + 1] - cs[c];
			int f = c == B2G_OVERFLOW ? 0 : res_first( n, rank, ctas );
			int l = c == B2G_OVERFLOW ? ( rank == 0 ? n : 0 ) : res_first( n, rank + 1, ctas );
			share[c].first = cs[c] + f;
			share[c].count = l - f;
			share[c].base = ONCHIP ? base : cs[c] + f;
			base += l - f;
		}
		s_ovSlots = 0;
	}
	__syncthreads();
	SmemRows m;
	if constexpr ( ONCHIP )
		m = res_carve_rows( smem, P.rowCap );
	else
		m = res_global_rows( W );
	const int rows = share[B2G_COLORS - 1].base + share[B2G_COLORS - 1].count;
	if constexpr ( ONCHIP )
		prepare_rows( W, m, rows, nullptr, nullptr, ResSource{ share, 0 }, tid, T, sc );
	else
		for ( int c = 0; c < B2G_COLORS; ++c )
			for ( int j = tid; j < share[c].count; j += T )
				res_prepare_global( W, m, share[c].first + j, sc );
	ResBodies rb;
	rb.st0 = rb.st1 = nullptr;
	rb.flags = rb.awake = nullptr;
	rb.term = smem + 9 * P.rowCap;
	rb.ad = (float*)( rb.term + P.bodyCap );
	const int af = res_first( P.awakeCount, rank, ctas );
	const int n = res_first( P.awakeCount, rank + 1, ctas ) - af;
	for ( int j = tid; j < n; j += T )
		res_terms( W, rb, j, W.awake[af + j], sc );
	const ResJoints J{};
	ResOverflow ov = res_carve_overflow( smem + P.ovOffset, P.ovOffset ? ovRows : 0, 0 );
	if ( rank == 0 && P.ovOffset )
	{
		__syncthreads();
		res_index_overflow<T, false>( ov, m, J, share[B2G_OVERFLOW], 0, ovRows, &s_ovSlots );
	}
	ResBarrier<0> bar{ ctl, ctas, 0u };
	bar.sync();
	L2Bodies G{ (float4*)W.state };
	res_run<0, T, false, false>( P, share, m, J, G, rb, (float4*)W.state, W.awake + af, n, bar, rank, sc, ov, s_ovSlots );
	if constexpr ( ONCHIP )
		store_impulses( W, m, rows, share[B2G_OVERFLOW].base, tid, T );
	else
		for ( int c = 0; c < B2G_COLORS; ++c )
		{
			const int f = share[c].base;
			const SmemRows part = { m.idx + f, m.nf + f, m.ms + f, m.anc0 + f, m.anc1 + f, m.coef0 + f, m.coef1 + f, m.imp0 + f, m.imp1 + f };
			store_impulses( W, part, share[c].count, c == B2G_OVERFLOW ? 0 : share[c].count, tid, T );
		}
	/* no CTA writes a state after its last barrier */
	if ( tid == 0 && grid_ended( ctl ) == ctas - 1 && *(volatile int*)( ctl + 2 ) != 0 )
		mark_lost( W, P.awakeCount, cs[B2G_COLORS] );
}

/* ------------------------------------------------------------------ host side */
#define RES_MAX_DEVICES 64
#define CLUSTER_THREADS 256
#define GRID_THREADS 256

typedef void ( *ResClusterKernel )( const b2gDevWorld, const ResidentPlan, const b2gStepConst );
typedef void ( *ResGridKernel )( const b2gDevWorld, const ResidentPlan, const b2gStepConst, int* );

struct ResDevice
{
	int looked; /* set last: the fields below do not change any more */
	int cluster; /* clusters of B2G_FUSED_CTAS CTAs can be launched */
	int sms;	 /* SMs of a cooperative launch, 0 when there is none */
};

static ResDevice s_devices[RES_MAX_DEVICES];

static cudaLaunchConfig_t res_config( cudaLaunchAttribute* attr, int ctas, int cluster, int threads, size_t smem, cudaStream_t s )
{
	cudaLaunchConfig_t cfg = {};
	cfg.gridDim = dim3( (unsigned)ctas, 1, 1 );
	cfg.blockDim = dim3( (unsigned)threads, 1, 1 );
	cfg.dynamicSmemBytes = smem;
	cfg.stream = s;
	cfg.attrs = attr;
	if ( cluster > 1 )
	{
		attr[0].id = cudaLaunchAttributeClusterDimension;
		attr[0].val.clusterDim.x = (unsigned)cluster;
		attr[0].val.clusterDim.y = 1;
		attr[0].val.clusterDim.z = 1;
		cfg.numAttrs = 1;
	}
	else if ( cluster == 0 )
	{
		attr[0].id = cudaLaunchAttributeCooperative;
		attr[0].val.cooperative = 1;
		cfg.numAttrs = 1;
	}
	return cfg;
}

template <class K>
static bool res_opt_in( K kernel, bool cluster )
{
	bool ok = cudaFuncSetAttribute( kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, RES_SMEM_MAX ) == cudaSuccess;
	if ( cluster )
		ok = cudaFuncSetAttribute( kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1 ) == cudaSuccess && ok;
	return ok;
}

/* What the current device can launch; looked up once per device (any number of threads
 * may look at once: they write the same values). */
static const ResDevice* res_device( void )
{
	int dev = 0;
	if ( cudaGetDevice( &dev ) != cudaSuccess || dev < 0 || dev >= RES_MAX_DEVICES )
		return nullptr;
	ResDevice* d = s_devices + dev;
	if ( __atomic_load_n( &d->looked, __ATOMIC_ACQUIRE ) )
		return d;
	int cluster = 0, sms = 0, coop = 0, blocks = 0;
	auto wide = k_solve_cluster<B2G_FUSED_CTAS, CLUSTER_THREADS>;
	bool ok = res_opt_in( k_solve_cluster<1, CLUSTER_THREADS>, false ) && res_opt_in( wide, true );
	if ( ok )
	{
		cudaLaunchAttribute attr[1];
		cudaLaunchConfig_t cfg = res_config( attr, B2G_FUSED_CTAS, B2G_FUSED_CTAS, CLUSTER_THREADS, RES_SMEM_MAX, nullptr );
		int n = 0;
		cluster = cudaOccupancyMaxActiveClusters( &n, wide, &cfg ) == cudaSuccess && n >= 1;
	}
	ok = res_opt_in( k_solve_grid<GRID_THREADS, true>, false ) && res_opt_in( k_solve_grid<GRID_THREADS, false>, false );
	cudaDeviceGetAttribute( &coop, cudaDevAttrCooperativeLaunch, dev );
	cudaDeviceGetAttribute( &sms, cudaDevAttrMultiProcessorCount, dev );
	if ( ok == false || coop == 0 ||
		 cudaOccupancyMaxActiveBlocksPerMultiprocessor( &blocks, k_solve_grid<GRID_THREADS, true>, GRID_THREADS, RES_SMEM_MAX ) != cudaSuccess || blocks < 1 )
		sms = 0;
	cudaGetLastError();
	d->cluster = cluster;
	d->sms = sms;
	__atomic_store_n( &d->looked, 1, __ATOMIC_RELEASE );
	return d;
}

/* Shared memory of CTA 0 with its overflow cache, which is left out when it does not fit. */
static size_t res_with_overflow( ResidentPlan* P, size_t bytes, int ovRows )
{
	P->ovOffset = 0;
	size_t at = ( bytes + 15 ) / 16;
	if ( ovRows > 0 && ovRows <= RES_OVERFLOW_MAX && 16 * at + res_overflow_bytes( ovRows, 0 ) <= RES_SMEM_MAX )
	{
		P->ovOffset = (int)at;
		bytes = 16 * at + res_overflow_bytes( ovRows, 0 );
	}
	return bytes;
}

/* The solver stage of caller buffers in one launch: the number of launches, 0 when this
 * device or set needs the per-phase kernels, or -1 on a launch error.  ctl: four ints of
 * device memory for a grid's barrier. */
extern "C" int b2gd_contact_resident( b2gDevWorld* w, const b2gSolvePlan* plan, const b2gStepConst* sc, int* ctl )
{
	const ResDevice* d = res_device();
	if ( d == nullptr )
		return 0;
	const int* cs = plan->colorStart;
	const int ovRows = cs[B2G_COLORS] - cs[B2G_OVERFLOW];
	ResidentPlan P;
	memset( &P, 0, sizeof( P ) );
	memcpy( P.colorStart, cs, sizeof( P.colorStart ) );
	memcpy( P.active, plan->active, sizeof( P.active ) );
	P.activeCount = plan->activeCount;
	P.awakeCount = plan->awakeCount;
	cudaStream_t s = (cudaStream_t)w->stream;
	cudaLaunchAttribute attr[1];

	/* One CTA, else a whole cluster, when it holds the set (res_body_cap).  One CTA is the
	 * faster one as long as it does (1200
	 * contacts: 58 us, 80 in a cluster); clusters of 2, 4 or 8 take what 16 take (2000
	 * contacts: 78 to 82 us), so there is no space between the two; a grid is slower
	 * wherever a cluster holds the set (20000 contacts: 201 us, 110 in a cluster). */
	const int spaces[] = { 1, B2G_FUSED_CTAS };
	for ( int ctas : spaces )
	{
		if ( ctas > 1 && d->cluster == 0 )
			break;
		P.bodyCap = res_body_cap( cs, P.awakeCount, ctas );
		if ( P.bodyCap == 0 )
			continue;
		P.rowCap = res_row_cap( cs, ctas );
		size_t rows = RES_ROW_BYTES * (size_t)P.rowCap;
		size_t bytes = rows + RES_BODY_BYTES * (size_t)P.bodyCap;
		if ( ctas > 1 )
			bytes = res_with_overflow( &P, bytes, ovRows );
		if ( ctas > 1 )
		{
			P.pushBytes = RES_SMEM_MAX - (int)rows;
			bytes = RES_SMEM_MAX;
		}
		auto kernel = ctas == 1 ? (ResClusterKernel)k_solve_cluster<1, CLUSTER_THREADS> : (ResClusterKernel)k_solve_cluster<B2G_FUSED_CTAS, CLUSTER_THREADS>;
		cudaLaunchConfig_t cfg = res_config( attr, ctas, ctas, CLUSTER_THREADS, bytes, s );
		return cudaLaunchKernelEx( &cfg, kernel, *w, P, *sc ) == cudaSuccess ? 1 : -1;
	}

	if ( d->sms == 0 )
		return 0;
	/* a grid: about 64 rows of the widest colour per CTA, so that small sets do not pay
	 * for the barrier of all SMs */
	int widest = 0;
	for ( int c = 0; c < B2G_OVERFLOW; ++c )
		widest = cs[c + 1] - cs[c] > widest ? cs[c + 1] - cs[c] : widest;
	int ctas = ( widest + 63 ) / 64;
	ctas = ctas < 1 ? 1 : ( ctas > d->sms ? d->sms : ctas );
	P.rowCap = res_row_cap( cs, ctas );
	P.bodyCap = ( ( P.awakeCount + ctas - 1 ) / ctas + 3 ) & ~3;
	size_t terms = 20u * (size_t)P.bodyCap;
	bool onChip = 144u * (size_t)P.rowCap + terms <= RES_SMEM_MAX;
	if ( onChip == false )
	{
		P.rowCap = 0;
		if ( terms > RES_SMEM_MAX )
			return 0;
	}
	if ( cudaMemsetAsync( ctl, 0, 4 * sizeof( int ), s ) != cudaSuccess )
		return -1;
	size_t bytes = res_with_overflow( &P, 144u * (size_t)P.rowCap + terms, ovRows );
	auto kernel = onChip ? (ResGridKernel)k_solve_grid<GRID_THREADS, true> : (ResGridKernel)k_solve_grid<GRID_THREADS, false>;
	cudaLaunchConfig_t cfg = res_config( attr, ctas, 0, GRID_THREADS, bytes, s );
	return cudaLaunchKernelEx( &cfg, kernel, *w, P, *sc, ctl ) == cudaSuccess ? 1 : -1;
}
