/*
 * fused.cu -- the whole solver stage of one world's step in one launch, by one CTA for a
 * small world, by a cluster of 16 CTAs for a larger one, and by a CTA per bin of islands
 * for a larger one whose islands are small (b2g_resident.h; why one launch, and what
 * bounds it, stands in resident.cu).
 *
 * Layout (dynamic shared memory of every CTA, rank r of CL):
 *   bodies  body ids are cut into CL contiguous blocks of bodyCap: body b lives in CTA
 *           b / bodyCap at slot b % bodyCap (the owner is found by a multiply-high with a
 *           host-computed reciprocal).  Every CTA has copies of the other bodies that its
 *           rows and joints touch and sends an update to the copy that is moved next
 *           (b2g_push.h); where the copies do not fit, or joints do not, rows
 *           reach a body of another CTA through distributed shared memory.
 *   rows    in a cluster the host groups each colour's rows by the CTA owning their first
 *           non-static body (rows of one colour share no body, so the order within a
 *           colour changes no result); CTA o holds rows [split[c][o], split[c][o+1]) of
 *           colour c as nine float4 arrays (structure of arrays, conflict-free).  Most
 *           body accesses of a row are then local.  The overflow colour's rows all live
 *           in CTA 0; thread 0 of CTA 0 solves them serially on the CTA's copies of
 *           their bodies.
 *   joints  CTA k takes an equal share of a colour's joints, in shared memory while they
 *           fit, else in the joint array; only one thread reads and writes a joint.
 *
 * Every CTA prepares its own rows and joints into shared memory: a staging kernel that
 * wrote the CTAs' images to global memory first took as long (large pyramid 116 us with
 * it, 117 without) and one launch more.
 *
 * Bound by the chain of about 113 dependent sweeps: a barrier and a row's own chain each.
 * Solver stage of a step before and after the one-CTA space and on-chip joints: pyramid of
 * 20 rows 97 -> 52 us, shape pile of 600 100 -> 68 us, 100 x 100 joint grid 421 -> 298 us.
 * With preparation and finalisation in the kernel: 47 us, 65 us; large pyramid 112 us, with
 * body copies 94, tumbler of 2000 370, with them 337 (83 to 95 overflow rows, one after the
 * other, 13 times a step: about 250 of it).  The joint grid's joints stay in L2 (5 us a
 * sweep); its stage runs beside the host's tree rebuild, which takes longer.
 */
#include "b2g_push.h"
#include "b2g_resident.h"

#include <string.h>

static_assert( RES_SMEM_MAX == B2G_BIN_BYTES_MAX && RES_JOINT_BYTES == B2G_BIN_JOINT_BYTES && RES_BODY_BYTES == B2G_BIN_BODY_BYTES,
			   "the host sizes what one CTA holds" );

/* 512 threads and 256 take the same time in the contact sweeps (large pyramid 117 us); joint
 * sweeps want the wider CTA (100 x 100 joint grid: solver stage 354 us with 256, 298 with
 * 512) */
#define FUSED_THREADS 512
#define FUSED_CLUSTER B2G_FUSED_CTAS

/* Rows of colour c owned by CTA o: [at[c][o], at[c][o + 1]) within the colour. */
struct FusedSplit
{
	int at[B2G_OVERFLOW][B2G_FUSED_CTAS + 1];
	unsigned bodyCapInv; /* ceil(2^32 / bodyCap), for the owner of a body id */
};

/* Islands share no constraint and no moving body, so bins of them are worlds of their
 * own to the solver.  Per bin BIN_INTS ints: row starts of the 12 colours and the end,
 * joint starts and end, first body and bodies; then the rows' contact ids, the joint ids
 * and the bodies' awake indices bin by bin, and every body id's slot in its bin.
 */
#define BIN_INTS B2G_BIN_INTS
struct FusedBins
{
	const int* table;
	const int* rows;
	const int* joints;
	const int* awake;
	const int* slot;
};

template <int CL, bool JOINTS, bool BINS = false>
__global__ void __launch_bounds__( FUSED_THREADS, 1 ) k_solve_world( const __grid_constant__ b2gDevWorld W, const __grid_constant__ ResidentPlan P,
																	 const __grid_constant__ FusedSplit S, const __grid_constant__ FusedBins bins,
																	 const __grid_constant__ b2gStepConst sc )
{
	/* bins of small islands are launched with fewer threads */
	const int T = BINS ? (int)blockDim.x : FUSED_THREADS;
	constexpr int CT = BINS ? 0 : FUSED_THREADS;
	const int* const bin = BINS ? bins.table + BIN_INTS * blockIdx.x : nullptr;
	const int* const rowList = BINS ? bins.rows : W.solveList;
	const int* const jointList = BINS ? bins.joints : W.jointList;
	extern __shared__ float4 smem[];
	__shared__ ResShare share[B2G_COLORS];
	__shared__ int s_rows, s_joints, s_awake, s_ovSlots;
	__shared__ PushShared push;
	cg::cluster_group cl = cg::this_cluster();
	const int rank = CL == 1 ? 0 : (int)cl.block_rank();
	const int tid = threadIdx.x;
	const int* cs = P.colorStart;
	const int* js = P.jointStart;
	SmemRows m = res_carve_rows( smem, P.rowCap );
	ResBodies rb = res_carve_bodies( smem + ( CL == 1 ? 9 * P.rowCap : P.bodyOffset ), P.bodyCap );
	float4* gst = (float4*)W.state;

	if ( tid < B2G_COLORS )
	{
		const bool ov = tid == B2G_OVERFLOW;
		const int n = cs[tid + 1] - cs[tid], nj = JOINTS ? js[tid + 1] - js[tid] : 0;
		int f, l, jf, jl;
		if ( BINS )
		{
			f = bin[tid] - cs[tid];
			l = bin[tid + 1] - cs[tid];
			jf = JOINTS ? bin[B2G_COLORS + 1 + tid] - js[tid] : 0;
			jl = JOINTS ? bin[B2G_COLORS + 2 + tid] - js[tid] : 0;
		}
		else if ( CL == 1 || ov )
		{
			const bool mine = rank == 0;
			f = jf = 0;
			l = mine ? n : 0;
			jl = mine ? nj : 0;
		}
		else
		{
			f = S.at[tid][rank];
			l = S.at[tid][rank + 1];
			jf = res_first( nj, rank, CL );
			jl = res_first( nj, rank + 1, CL );
		}
		share[tid].first = cs[tid] + f;
		share[tid].count = l - f;
		share[tid].jfirst = js[tid] + jf;
		share[tid].jcount = jl - jf;
	}
	if ( tid == 0 )
		s_awake = s_ovSlots = 0;
	__syncthreads();
	if ( tid == 0 )
	{
		int base = 0, jbase = 0;
		for ( int c = 0; c < B2G_COLORS; ++c )
		{
			share[c].base = base;
			share[c].jbase = jbase;
			base += share[c].count;
			jbase += share[c].jcount;
		}
		s_rows = base;
		s_joints = jbase;
	}
	__syncthreads();
	const int rows = s_rows, colourRows = share[B2G_OVERFLOW].base;
	/* one CTA: awake bodies in list order, their awake indices kept for finalisation; a
	 * cluster: the block of ids that this CTA owns */
	int bodies = P.awakeCount;
	if ( BINS )
		bodies = bin[BIN_INTS - 1];
	if ( CL > 1 )
	{
		bodies = P.bodyIdCount - rank * P.bodyCap;
		bodies = bodies < 0 ? 0 : ( bodies > P.bodyCap ? P.bodyCap : bodies );
	}
	auto load_owned = [&]() {
		const int first = rank * P.bodyCap;
		for ( int s = tid; s < bodies; s += T )
		{
			rb.st0[s] = gst[2 * ( first + s )];
			rb.st1[s] = gst[2 * ( first + s ) + 1];
			rb.flags[s] = -1;
		}
		__syncthreads();
		/* the awake bodies among them, with their awake indices; four of the list at a
		 * time, and the terms behind it: one round trip each */
		constexpr int U = 4;
		for ( int i0 = tid; i0 < P.awakeCount; i0 += U * T )
		{
			int s[U];
#pragma unroll
			for ( int u = 0; u < U; ++u )
				s[u] = i0 + u * T < P.awakeCount ? W.awake[i0 + u * T] - first : -1;
#pragma unroll
			for ( int u = 0; u < U; ++u )
				if ( s[u] >= 0 && s[u] < bodies )
				{
					rb.awake[atomicAdd( &s_awake, 1 )] = s[u];
					rb.flags[s[u]] = i0 + u * T;
				}
		}
		__syncthreads();
		for ( int j = tid; j < s_awake; j += T )
			res_terms( W, rb, rb.awake[j], first + rb.awake[j], sc );
	};
	PushBodies PB;
	if constexpr ( CL == 1 )
	{
		const int* mine = BINS ? bins.awake + bin[BIN_INTS - 2] : nullptr;
		for ( int j = tid; j < bodies; j += T )
		{
			const int i = BINS ? mine[j] : j;
			const int b = W.awake[i];
			const int s = BINS ? j : b;
			rb.awake[j] = s;
			rb.flags[j] = i;
			rb.st0[s] = gst[2 * b];
			rb.st1[s] = gst[2 * b + 1];
			res_terms( W, rb, s, b, sc );
		}
		if ( tid == 0 )
			s_awake = bodies;
	}
	else
	{
		if ( P.pushCap > 0 )
		{
			push_carve( smem + P.bodyOffset, P.pushCap, P.bodyCap, rank, PB, rb );
			push_init( PB, push, P, P.bodyCap );
		}
		load_owned();
	}
	/* The narrowphase, which this launch may overlap up to here: nothing above reads what it
	 * writes, and nothing above writes to global memory.  With events in it the host solves
	 * on other lists; every CTA takes the same branch: no barrier is left waiting. */
	asm volatile( "griddepcontrol.wait;" ::: "memory" );
	if ( W.guardEvents && __ldcg( W.counters ) != 0 )
		return;
	ResJoints J;
	J.local = JOINTS && P.jointCap > 0 ? (char*)( smem + P.jointOffset ) : nullptr;
	J.array = W.joints;
	J.list = jointList;
	if ( JOINTS && J.local != nullptr )
	{
		for ( int t = tid, c = 0; t < 64 * s_joints; t += T )
		{
			const int k = t >> 6;
			while ( k >= share[c].jbase + share[c].jcount )
				++c;
			const int id = jointList[share[c].jfirst + ( k - share[c].jbase )];
			( (int*)J.local )[RES_JOINT_WORDS * k + ( t & 63 )] = ( (const int*)( W.joints + id ) )[t & 63];
		}
	}
	prepare_rows( W, m, rows, rowList, BINS ? bins.slot : nullptr, ResSource{ share, 0 }, tid, T, sc );
	if ( JOINTS )
	{
		__syncthreads();
		for ( int k = tid, c = 0; k < s_joints; k += T )
		{
			while ( k >= share[c].jbase + share[c].jcount )
				++c;
			b2gJointDev* j = J.at( share[c].jfirst, share[c].jbase, k - share[c].jbase );
			prepare_joint_at( W, j, sc );
			if ( BINS )
			{
				j->indexA = j->indexA >= 0 ? bins.slot[j->indexA] : -1;
				j->indexB = j->indexB >= 0 ? bins.slot[j->indexB] : -1;
			}
		}
	}
	ResBarrier<CL> bar{ nullptr, CL, 0 };
	bool pushes = false;
	int* const ovList = rb.awake + P.bodyCap;
	if constexpr ( CL > 1 )
	{
		if ( P.pushCap > 0 )
		{
			pushes = push_exchange<JOINTS>( cl, PB, push, P.pushCap, P.bodyCap, S.bodyCapInv, rows, s_joints, share, m, J, ovList,
											rb, s_awake, [&]( int s ) { return rb.flags[s] >= 0; } );
			if ( pushes == false )
			{
				/* more copies than a CTA can hold: states in their owners' CTAs only */
				rb = res_carve_bodies( smem + P.bodyOffset, P.bodyCap );
				if ( tid == 0 )
					s_awake = 0;
				__syncthreads();
				load_owned();
			}
		}
	}
	const int ovRows = cs[B2G_COLORS] - cs[B2G_OVERFLOW], ovJoints = JOINTS ? js[B2G_COLORS] - js[B2G_OVERFLOW] : 0;
	ResOverflow ov = res_carve_overflow( smem + P.ovOffset, P.ovOffset ? ovRows : 0, P.ovOffset ? ovJoints : 0 );
	if ( CL > 1 && rank == 0 && P.ovOffset && pushes == false )
	{
		__syncthreads();
		res_index_overflow<CT, JOINTS>( ov, m, J, share[B2G_OVERFLOW], ovJoints, ovRows, &s_ovSlots );
	}
	bar.sync();
	const int awake = s_awake;
	if constexpr ( CL == 1 )
	{
		LocalBodies B;
		B.st0 = rb.st0;
		B.st1 = rb.st1;
		res_run<CL, CT, true, JOINTS, BINS>( P, share, m, J, B, rb, gst, nullptr, awake, bar, rank, sc, ov, s_ovSlots );
	}
	else if ( pushes )
		push_run<CT, JOINTS>( P, share, m, J, PB, push, rb, awake, push.copies - P.bodyCap, ovList, sc );
	else
	{
		DsmemBodies B{ { cl, rb.st0, rb.st1, P.bodyCap, rank, S.bodyCapInv } };
		res_run<CL, CT, true, JOINTS>( P, share, m, J, B, rb, gst, nullptr, awake, bar, rank, sc, ov, s_ovSlots );
	}

	store_impulses( W, m, rows, colourRows, tid, T );
	if ( JOINTS && J.local != nullptr )
	{
		for ( int t = tid, c = 0; t < 64 * s_joints; t += T )
		{
			const int k = t >> 6;
			while ( k >= share[c].jbase + share[c].jcount )
				++c;
			const int id = jointList[share[c].jfirst + ( k - share[c].jbase )];
			( (int*)( W.joints + id ) )[t & 63] = ( (const int*)J.local )[RES_JOINT_WORDS * k + ( t & 63 )];
		}
	}

	/* finalisation (reference src/solver.c:165-351) of the bodies whose states are here,
	 * then the counts of its records and sleepy bodies to the host */
	for ( int j = tid; j < awake; j += T )
	{
		const int s = rb.awake[j], i = CL == 1 ? rb.flags[j] : rb.flags[s];
		const int b = CL == 1 ? W.awake[i] : rank * P.bodyCap + s;
		gst[2 * b] = rb.st0[s];
		finalize_state( W, i, b, rb.st0[s], rb.st1[s], sc );
	}
	if ( pushes == false )
		bar.sync();
	else if ( push_end( cl, push ) && tid == 0 )
		W.hostCounters[2] = 1;
	if ( rank == 0 && tid == 0 )
	{
		bool last = true;
		if ( BINS )
		{
			__threadfence();
			last = atomicAdd( W.counters + 2, 1 ) == (int)gridDim.x - 1;
			__threadfence();
		}
		if ( last )
		{
			W.hostCounters[1] = __ldcg( W.counters + 1 );
			W.hostCounters[3] = __ldcg( W.counters + 3 );
			/* every CTA has passed the guard: the next narrowphase starts from zero */
			W.counters[0] = W.counters[1] = W.counters[2] = W.counters[3] = 0;
		}
	}
}

static_assert( sizeof( b2gJointDev ) == 256, "the joint copies move 64 words" );

typedef void ( *FusedKernel )( const b2gDevWorld, const ResidentPlan, const FusedSplit, const FusedBins, const b2gStepConst );

/* early: the launch follows the narrowphase directly and may start beside it, up to the
 * kernel's griddepcontrol.wait. */
static cudaLaunchConfig_t fused_config( cudaLaunchAttribute* attr, int ctas, size_t smem, cudaStream_t stream, bool early, int grid = 0,
										int threads = FUSED_THREADS )
{
	cudaLaunchConfig_t cfg = {};
	cfg.gridDim = dim3( (unsigned)( grid > 0 ? grid : ctas ), 1, 1 );
	cfg.blockDim = dim3( (unsigned)threads, 1, 1 );
	cfg.dynamicSmemBytes = smem;
	cfg.stream = stream;
	cfg.attrs = attr;
	if ( ctas > 1 )
	{
		attr[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
		attr[cfg.numAttrs].val.clusterDim.x = (unsigned)ctas;
		attr[cfg.numAttrs].val.clusterDim.y = 1;
		attr[cfg.numAttrs].val.clusterDim.z = 1;
		cfg.numAttrs += 1;
	}
	if ( early )
	{
		attr[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
		attr[cfg.numAttrs].val.programmaticStreamSerializationAllowed = 1;
		cfg.numAttrs += 1;
	}
	return cfg;
}

/* Whether clusters of FUSED_CLUSTER CTAs can be launched on the current device; the
 * kernels' attributes are set on the first look. */
static int fused_cluster_ready( void )
{
	/* per device: 0 unknown, 1 available, -1 unavailable */
	static int s_readyByDevice[64];
	int dev = 0;
	if ( cudaGetDevice( &dev ) != cudaSuccess || dev < 0 || dev >= 64 )
		return -1;
	int ready = __atomic_load_n( s_readyByDevice + dev, __ATOMIC_ACQUIRE );
	if ( ready != 0 )
		return ready;
	bool ok = true;
	for ( FusedKernel k : { k_solve_world<1, false>, k_solve_world<1, true>, k_solve_world<1, false, true>, k_solve_world<1, true, true> } )
		ok = ok && cudaFuncSetAttribute( k, cudaFuncAttributeMaxDynamicSharedMemorySize, RES_SMEM_MAX ) == cudaSuccess;
	for ( FusedKernel k : { k_solve_world<FUSED_CLUSTER, false>, k_solve_world<FUSED_CLUSTER, true> } )
	{
		ok = ok && cudaFuncSetAttribute( k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1 ) == cudaSuccess &&
			 cudaFuncSetAttribute( k, cudaFuncAttributeMaxDynamicSharedMemorySize, RES_SMEM_MAX ) == cudaSuccess;
		cudaLaunchAttribute attr[2];
		cudaLaunchConfig_t cfg = fused_config( attr, FUSED_CLUSTER, RES_SMEM_MAX, nullptr, false );
		int clusters = 0;
		ok = ok && cudaOccupancyMaxActiveClusters( &clusters, k, &cfg ) == cudaSuccess && clusters >= 1;
	}
	cudaGetLastError();
	ready = ok ? 1 : -1;
	__atomic_store_n( s_readyByDevice + dev, ready, __ATOMIC_RELEASE );
	return ready;
}

/* Launches the fused solver and finalisation when the world fits on chip; returns the number of launches,
 * 0 when it does not fit (or clusters of FUSED_CLUSTER CTAs are unavailable) and the
 * caller must use the per-phase kernels, or -1 on a launch error. */
extern "C" int b2gd_solver_fused( b2gDevWorld* w, const b2gSolvePlan* plan, const b2gStepConst* sc )
{
	if ( plan->bodyIdCount <= 0 || plan->bodyBlock <= 0 || fused_cluster_ready() != 1 )
		return 0;
	const int* cs = plan->colorStart;
	const int* js = plan->jointStart;
	const int joints = js[B2G_COLORS];
	/* launched behind the narrowphase, whose kernel was the last on the stream: the CTAs
	 * then load their bodies beside it (large pyramid 131.8 -> 127 us a step with its read,
	 * shape pile 88.3 -> 83.4) */
	const bool early = w->guardEvents && w->collideLast && w->timing == 0;
	const int ovR = cs[B2G_COLORS] - cs[B2G_OVERFLOW], ovJ = js[B2G_COLORS] - js[B2G_OVERFLOW];
	ResidentPlan P;
	FusedSplit S;
	FusedBins bins = {};
	memset( &P, 0, sizeof( P ) );
	memset( &S, 0, sizeof( S ) );
	memcpy( P.colorStart, cs, sizeof( P.colorStart ) );
	memcpy( P.jointStart, js, sizeof( P.jointStart ) );
	memcpy( P.active, plan->active, sizeof( P.active ) );
	P.activeCount = plan->activeCount;
	P.awakeCount = plan->awakeCount;
	P.bodyIdCount = plan->bodyIdCount;

	/* one CTA when it holds the world, joints included: no barrier crosses SMs (0.45 us a
	 * sweep for the 20-row pyramid, 0.85 us in a cluster) */
	size_t one = b2g_bin_bytes( cs[B2G_COLORS], plan->bodyIdCount, 0 );
	if ( b2g_bin_bytes( cs[B2G_COLORS], plan->bodyIdCount, joints ) <= RES_SMEM_MAX )
	{
		P.rowCap = cs[B2G_COLORS] > 0 ? cs[B2G_COLORS] : 1;
		P.bodyCap = ( plan->bodyIdCount + 3 ) & ~3;
		P.jointCap = joints;
		P.jointOffset = (int)( one / 16 );
		cudaLaunchAttribute attr[2];
		cudaLaunchConfig_t cfg = fused_config( attr, 1, one + RES_JOINT_BYTES * (size_t)joints, (cudaStream_t)w->stream, early );
		FusedKernel k = joints > 0 ? k_solve_world<1, true> : k_solve_world<1, false>;
		return cudaLaunchKernelEx( &cfg, k, *w, P, S, bins, *sc ) == cudaSuccess ? 1 : -1;
	}

	if ( plan->binCount > 0 )
	{
		/* a CTA per bin: 128 threads cover the widest colour of small islands, and leave
		 * room for several CTAs on an SM */
		const int* at = w->bins;
		bins.table = at;
		bins.rows = at + BIN_INTS * plan->binCount;
		bins.joints = bins.rows + cs[B2G_COLORS];
		bins.awake = bins.joints + joints;
		bins.slot = bins.awake + plan->awakeCount;
		P.rowCap = plan->binRows > 0 ? plan->binRows : 1;
		P.bodyCap = ( plan->binBodies + 3 ) & ~3;
		P.jointCap = plan->binJoints;
		size_t bytes = b2g_bin_bytes( plan->binRows, plan->binBodies, 0 );
		P.jointOffset = (int)( bytes / 16 );
		cudaLaunchAttribute attr[2];
		cudaLaunchConfig_t cfg = fused_config( attr, 1, bytes + RES_JOINT_BYTES * (size_t)plan->binJoints, (cudaStream_t)w->stream, early, plan->binCount,
											   plan->binWidest <= 128 ? 128 : FUSED_THREADS );
		FusedKernel k = joints > 0 ? k_solve_world<1, true, true> : k_solve_world<1, false, true>;
		return cudaLaunchKernelEx( &cfg, k, *w, P, S, bins, *sc ) == cudaSuccess ? 1 : -1;
	}

	/* body ids and slots below 2^16: the owner division is one multiply-high */
	if ( plan->bodyIdCount >= 65536 )
		return 0;
	const int CL = FUSED_CLUSTER;
	P.bodyCap = plan->bodyBlock;
	S.bodyCapInv = P.bodyCap > 1 ? (unsigned)( ( ( 1ull << 32 ) + (unsigned long long)P.bodyCap - 1 ) / (unsigned long long)P.bodyCap ) : 0u;
	int perCta[B2G_FUSED_CTAS] = { ovR };
	for ( int c = 0; c < B2G_OVERFLOW; ++c )
	{
		int n = 0;
		for ( int o = 0; o < CL; ++o )
		{
			S.at[c][o] = n;
			n += plan->rowSplit[c][o];
			perCta[o] += plan->rowSplit[c][o];
		}
		S.at[c][CL] = n;
		if ( n != cs[c + 1] - cs[c] )
			return 0; /* rows not grouped by owner */
		P.jointCap += ( js[c + 1] - js[c] + CL - 1 ) / CL;
	}
	P.jointCap += ovJ;
	P.rowCap = 1;
	for ( int o = 0; o < CL; ++o )
		P.rowCap = perCta[o] > P.rowCap ? perCta[o] : P.rowCap;
	/* rows, joints while they fit, then the bodies with the overflow cache or, in their
	 * place, the copies of push_run: as many as there is room for */
	const size_t rowBytes = 144u * (size_t)P.rowCap;
	const size_t bodyBytes = ( RES_BODY_BYTES * (size_t)P.bodyCap + 15 ) / 16 * 16;
	size_t bytes = rowBytes + bodyBytes;
	if ( bytes > RES_SMEM_MAX )
		return 0;
	size_t ovBytes = 0;
	if ( ovR + ovJ > 0 && ovR + ovJ <= RES_OVERFLOW_MAX && bytes + res_overflow_bytes( ovR, ovJ ) <= RES_SMEM_MAX )
		ovBytes = ( res_overflow_bytes( ovR, ovJ ) + 15 ) / 16 * 16;
	bytes += ovBytes;
	size_t jointBytes = ( RES_JOINT_BYTES * (size_t)P.jointCap + 15 ) / 16 * 16;
	if ( bytes + jointBytes <= RES_SMEM_MAX )
		P.jointOffset = (int)( rowBytes / 16 );
	else
	{
		P.jointCap = 0;
		jointBytes = 0;
	}
	bytes += jointBytes;
	P.bodyOffset = (int)( ( rowBytes + jointBytes ) / 16 );
	if ( ovBytes > 0 )
		P.ovOffset = P.bodyOffset + (int)( bodyBytes / 16 );
	const size_t fixed = rowBytes + jointBytes + PUSH_OWNED_BYTES * (size_t)P.bodyCap + 8u * (size_t)( ovR + ovJ );
	if ( ( joints == 0 || jointBytes > 0 ) && fixed + PUSH_COPY_BYTES * (size_t)P.bodyCap <= RES_SMEM_MAX )
	{
		size_t cap = ( RES_SMEM_MAX - fixed ) / PUSH_COPY_BYTES;
		P.pushCap = cap < (size_t)P.bodyIdCount ? (int)cap : P.bodyIdCount;
		P.pushCap = P.pushCap < P.bodyCap ? P.bodyCap : P.pushCap;
		const size_t need = fixed + PUSH_COPY_BYTES * (size_t)P.pushCap;
		bytes = need > bytes ? need : bytes;
	}
	cudaLaunchAttribute attr[2];
	cudaLaunchConfig_t cfg = fused_config( attr, CL, bytes, (cudaStream_t)w->stream, early );
	FusedKernel k = joints > 0 ? k_solve_world<FUSED_CLUSTER, true> : k_solve_world<FUSED_CLUSTER, false>;
	return cudaLaunchKernelEx( &cfg, k, *w, P, S, bins, *sc ) == cudaSuccess ? 1 : -1;
}
