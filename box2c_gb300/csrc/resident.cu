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
 *             that solves them, body b in CTA b / block, reached through distributed
 *             shared memory; hardware cluster barriers.
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
 * a colour, where shared-memory bandwidth shows), 0.75 to 1 us in a cluster, 2 us in a
 * grid (an L2 round trip to arrive and one to see it).  b2SolveContacts, one kernel per
 * phase before and one resident kernel now, four substeps: 900 contacts 420 -> 52 us (a
 * cluster takes 82), 15000 420 -> 102 (a grid takes 199), 60000 424 -> 207; with 17
 * overflow rows at 15000 contacts 799 -> 185.
 */
#include "b2g_cluster.h"
#include "b2g_device.h"

#include <cuda_runtime.h>

#include <string.h>

/* dynamic shared memory per CTA, leaving 1 KB of the 227 KB opt-in limit for statics */
#define RES_SMEM_MAX ( 226 * 1024 )
#define RES_OVERFLOW_MAX 512
/* polls of a grid barrier before it gives up (seconds; a cooperative launch never gets
 * there) */
#define RES_SPIN_LIMIT ( 1 << 22 )

struct ResidentPlan
{
	int colorStart[B2G_COLORS + 1];
	int active[B2G_COLORS];
	int activeCount;
	int awakeCount;
	int ctas;
	int rowCap;	 /* row slots per CTA (0: rows in the row arrays) */
	int bodyCap; /* body slots per CTA in shared memory; a grid's velocity-term slots */
	int ovOffset; /* float4 offset of the overflow cache, 0 without one */
};

/* Overflow cache of CTA 0: for R overflow rows with E = 2 R body ends, the rows' indices
 * with body slots (int4 x R), slot states (2 x float4 x E), slot bodies, first occurrences
 * and slots per end (3 x int x E). */
struct ResOverflow
{
	int4* idx;
	float4* st0;
	float4* st1;
	int* body;
	int* first;
	int* slot;
};

static __host__ __device__ size_t res_overflow_bytes( int R ) { return 16u * 5u * (size_t)R + 24u * (size_t)R; }

__device__ __forceinline__ ResOverflow res_carve_overflow( float4* base, int R )
{
	int E = 2 * R;
	ResOverflow o;
	o.idx = (int4*)base;
	o.st0 = base + R;
	o.st1 = o.st0 + E;
	o.body = (int*)( o.st1 + E );
	o.first = o.body + E;
	o.slot = o.first + E;
	return o;
}

/* Bytes of one body slot in shared memory: two state float4, the velocity terms (float4
 * and float), flags and an entry of the awake list. */
#define RES_BODY_BYTES 60

struct ResBodies
{
	float4* st0;  /* v.x v.y w tag */
	float4* st1;  /* dp.x dp.y dq.c dq.s */
	float4* term; /* lvd.x lvd.y avd ld */
	float* ad;	  /* angular damping factor */
	int* flags;	  /* RES_AWAKE, RES_TOUCHED */
	int* awake;	  /* local awake slots */
};

enum
{
	RES_AWAKE = 1,
	RES_TOUCHED = 2,
};

__device__ __forceinline__ ResBodies res_carve_bodies( float4* base, int cap )
{
	ResBodies b;
	b.st0 = base;
	b.st1 = base + cap;
	b.term = base + 2 * cap;
	b.ad = (float*)( base + 3 * cap );
	b.flags = (int*)( b.ad + cap );
	b.awake = b.flags + cap;
	return b;
}

__device__ __forceinline__ SmemRows res_carve_rows( float4* base, int n )
{
	SmemRows m;
	m.idx = (int4*)base;
	m.nf = base + n;
	m.ms = base + 2 * n;
	m.anc0 = base + 3 * n;
	m.anc1 = base + 4 * n;
	m.coef0 = base + 5 * n;
	m.coef1 = base + 6 * n;
	m.imp0 = base + 7 * n;
	m.imp1 = base + 8 * n;
	return m;
}

__device__ __forceinline__ SmemRows res_global_rows( const b2gDevWorld& W )
{
	SmemRows m;
	m.idx = (int4*)W.kIdx;
	m.nf = (float4*)W.kNF;
	m.ms = (float4*)W.kMass;
	m.anc0 = (float4*)W.kAnchor[0];
	m.anc1 = (float4*)W.kAnchor[1];
	m.coef0 = (float4*)W.kCoef[0];
	m.coef1 = (float4*)W.kCoef[1];
	m.imp0 = (float4*)W.kImp[0];
	m.imp1 = (float4*)W.kImp[1];
	return m;
}

/* Body states in global memory, read and written at L2: other CTAs change them between
 * sweeps. */
struct L2Bodies
{
	float4* st;
	__device__ __forceinline__ DevState load( int b ) const
	{
		return b < 0 ? identity_state() : state_of( __ldcg( st + 2 * b ), __ldcg( st + 2 * b + 1 ) );
	}
	__device__ __forceinline__ DevState load_velocity( int b ) const
	{
		return b < 0 ? identity_state() : state_of( __ldcg( st + 2 * b ), make_float4( 0.0f, 0.0f, 1.0f, 0.0f ) );
	}
	__device__ __forceinline__ void store( int b, const DevState& x ) const
	{
		if ( b >= 0 )
			__stcg( st + 2 * b, velocity_word( x ) );
	}
	__device__ __forceinline__ float4 word0( int b ) const { return __ldcg( st + 2 * b ); }
	__device__ __forceinline__ float4 word1( int b ) const { return __ldcg( st + 2 * b + 1 ); }
	__device__ __forceinline__ void set_word0( int b, float4 v ) const { __stcg( st + 2 * b, v ); }
};

/* ClusterBodies with the words the overflow cache copies. */
struct DsmemBodies : ClusterBodies
{
	__device__ __forceinline__ float4 word0( int b ) const { return *word( st0, b ); }
	__device__ __forceinline__ float4 word1( int b ) const { return *word( st1, b ); }
	__device__ __forceinline__ void set_word0( int b, float4 v ) const { *word( st0, b ) = v; }
};

/* The one-CTA space's bodies are already local: the overflow pass needs no cache. */
struct LocalBodies : SharedBodies
{
	__device__ __forceinline__ float4 word0( int b ) const { return st0[b]; }
	__device__ __forceinline__ float4 word1( int b ) const { return st1[b]; }
	__device__ __forceinline__ void set_word0( int b, float4 v ) const { st0[b] = v; }
};

/* Barrier between sweeps.  A grid's barrier counts arrivals in ctl[0]; ctl[2] tells every
 * CTA that one gave up, after which no CTA waits again. */
template <int CL>
struct ResBarrier
{
	int* ctl;
	int ctas;
	unsigned target;
	__device__ __forceinline__ void sync()
	{
		if constexpr ( CL == 1 )
			__syncthreads();
		else if constexpr ( CL > 1 )
			cg::this_cluster().sync();
		else
		{
			__syncthreads();
			target += (unsigned)ctas;
			if ( threadIdx.x == 0 )
			{
				unsigned* count = (unsigned*)ctl;
				asm volatile( "red.release.gpu.global.add.u32 [%0], 1;" ::"l"( count ) : "memory" );
				int left = RES_SPIN_LIMIT;
				unsigned seen;
				do
				{
					asm volatile( "ld.acquire.gpu.global.u32 %0, [%1];" : "=r"( seen ) : "l"( count ) : "memory" );
				} while ( (int)( seen - target ) < 0 && --left > 0 && ( ( left & 1023 ) != 0 || *(volatile int*)( ctl + 2 ) == 0 ) );
				if ( (int)( seen - target ) < 0 )
					*(volatile int*)( ctl + 2 ) = 1;
			}
			__syncthreads();
		}
	}
};

struct ResShare
{
	int first, count, base; /* of one colour: rows [first, first + count) at local index base */
};

__device__ __forceinline__ int res_first( int n, int k, int ctas ) { return (int)( (long long)n * k / ctas ); }

/* One stage over all colours: the overflow set first (serially, CTA 0), then each active
 * colour with a barrier after it. */
template <int CL, int PHASE, int T, class Bodies>
__device__ __forceinline__ void res_stage( const ResidentPlan& P, const ResShare* share, const SmemRows& m, const Bodies& B,
										   ResBarrier<CL>& bar, int rank, const b2gStepConst& sc, const ResOverflow& ov, int ovSlots )
{
	const int* cs = P.colorStart;
	const int R = cs[B2G_COLORS] - cs[B2G_OVERFLOW];
	if ( R > 0 )
	{
		if ( rank == 0 )
		{
			const int base = share[B2G_OVERFLOW].base;
			if ( CL != 1 && P.ovOffset != 0 )
			{
				/* the set's bodies to local slots, the serial pass on them, velocities back:
				 * nothing else touches a body while the set runs */
				for ( int s = threadIdx.x; s < ovSlots; s += T )
				{
					int b = ov.body[s];
					ov.st0[s] = B.word0( b );
					ov.st1[s] = B.word1( b );
				}
				__syncthreads();
				if ( threadIdx.x == 0 )
				{
					SharedBodies OB{ ov.st0, ov.st1 };
					SmemRows mo = { ov.idx, m.nf + base, m.ms + base, m.anc0 + base, m.anc1 + base, m.coef0 + base, m.coef1 + base, m.imp0 + base, m.imp1 + base };
					for ( int i = 0; i < R; ++i )
						row_step( mo, OB, i, PHASE, true, sc );
				}
				__syncthreads();
				for ( int s = threadIdx.x; s < ovSlots; s += T )
					B.set_word0( ov.body[s], ov.st0[s] );
			}
			else if ( threadIdx.x == 0 )
			{
				for ( int i = 0; i < R; ++i )
					row_step( m, B, base + i, PHASE, true, sc );
			}
		}
		bar.sync();
	}
	if ( PHASE == F_WARM && sc.enableWarmStarting == 0 )
		return;
	for ( int a = 0; a < P.activeCount; ++a )
	{
		const ResShare s = share[P.active[a]];
		for ( int j = threadIdx.x; j < s.count; j += T )
			row_step( m, B, s.base + j, PHASE, false, sc );
		bar.sync();
	}
}

/* All substeps over bodies B.  Integration runs over this CTA's awake bodies: with states
 * in shared memory slots b.awake[0 .. awake), in global memory the ids list[0 .. awake). */
template <int CL, int T, bool SHARED_STATES, class Bodies>
__device__ __forceinline__ void res_run( const ResidentPlan& P, const ResShare* share, const SmemRows& m, const Bodies& B,
										 const ResBodies& rb, float4* gst, const int* list, int awake, ResBarrier<CL>& bar, int rank,
										 const b2gStepConst& sc, const ResOverflow& ov, int ovSlots )
{
	for ( int sub = 0; sub < sc.subSteps; ++sub )
	{
		for ( int j = threadIdx.x; j < awake; j += T )
		{
			const int s = SHARED_STATES ? rb.awake[j] : list[j];
			const int k = SHARED_STATES ? s : j;
			float4* p = SHARED_STATES ? rb.st0 + s : gst + 2 * s;
			DevState x = state_of( SHARED_STATES ? *p : __ldcg( p ), make_float4( 0.0f, 0.0f, 1.0f, 0.0f ) );
			float4 t4 = rb.term[k];
			VelocityTerms t;
			t.lvd = gv( t4.x, t4.y );
			t.avd = t4.z;
			t.ld = t4.w;
			t.ad = rb.ad[k];
			integrate_velocity( x, t, sc );
			if ( SHARED_STATES )
				*p = velocity_word( x );
			else
				__stcg( p, velocity_word( x ) );
		}
		bar.sync();
		res_stage<CL, F_WARM, T>( P, share, m, B, bar, rank, sc, ov, ovSlots );
		res_stage<CL, F_SOLVE, T>( P, share, m, B, bar, rank, sc, ov, ovSlots );
		for ( int j = threadIdx.x; j < awake; j += T )
		{
			const int s = SHARED_STATES ? rb.awake[j] : list[j];
			float4* p0 = SHARED_STATES ? rb.st0 + s : gst + 2 * s;
			float4* p1 = SHARED_STATES ? rb.st1 + s : gst + 2 * s + 1;
			DevState x = state_of( SHARED_STATES ? *p0 : __ldcg( p0 ), SHARED_STATES ? *p1 : __ldcg( p1 ) );
			integrate_position( x, sc.h );
			float4 v = make_float4( x.dp.x, x.dp.y, x.dq.c, x.dq.s );
			if ( SHARED_STATES )
				*p1 = v;
			else
				__stcg( p1, v );
		}
		bar.sync();
		res_stage<CL, F_RELAX, T>( P, share, m, B, bar, rank, sc, ov, ovSlots );
	}
	res_stage<CL, F_RESTITUTION, T>( P, share, m, B, bar, rank, sc, ov, ovSlots );
}

/* Overflow cache: the distinct bodies of the set's ends get slots in end order. */
template <int T>
__device__ __forceinline__ void res_index_overflow( const ResOverflow& ov, const SmemRows& m, int base, int R, int* slots )
{
	const int E = 2 * R;
	auto end_body = [&]( int e ) {
		int4 ix = m.idx[base + ( e >> 1 )];
		return ( e & 1 ) ? ix.y : ix.x;
	};
	for ( int e = threadIdx.x; e < E; e += T )
	{
		int b = end_body( e );
		int f = -1;
		if ( b >= 0 )
		{
			f = e;
			for ( int e2 = 0; e2 < e; ++e2 )
			{
				if ( end_body( e2 ) == b )
				{
					f = e2;
					break;
				}
			}
		}
		ov.first[e] = f;
	}
	__syncthreads();
	if ( threadIdx.x == 0 )
	{
		int K = 0;
		for ( int e = 0; e < E; ++e )
		{
			if ( ov.first[e] == e )
			{
				ov.slot[e] = K;
				ov.body[K++] = end_body( e );
			}
		}
		*slots = K;
	}
	__syncthreads();
	for ( int e = threadIdx.x; e < E; e += T )
	{
		int f = ov.first[e];
		int s = f < 0 ? -1 : ov.slot[f];
		int r = e >> 1;
		if ( e & 1 )
			ov.idx[r].y = s;
		else
		{
			int4 ix = m.idx[base + r];
			ov.idx[r].x = s;
			ov.idx[r].z = ix.z;
			ov.idx[r].w = ix.w;
		}
	}
}

/* Preparation of one row into m (reference src/contact_solver.c:597-808, :21-147). */
__device__ __forceinline__ int2 res_prepare( const b2gDevWorld& W, const SmemRows& m, int k, int local, const b2gStepConst& sc )
{
	const float4* gst = (const float4*)W.state;
	const float4* mass = (const float4*)W.mass;
	const float4 zero = make_float4( 0.0f, 0.0f, 0.0f, 0.0f );
	int cid = W.solveList ? W.solveList[k] : k;
	int ia = W.cBodies[2 * cid];
	int ib = W.cBodies[2 * cid + 1];
	DevState sA = ia >= 0 ? state_of( gst[2 * ia], gst[2 * ia + 1] ) : identity_state();
	DevState sB = ib >= 0 ? state_of( gst[2 * ib], gst[2 * ib + 1] ) : identity_state();
	Row r;
	prepare_row( r, W.manifold + cid, ia, ib, ia >= 0 ? mass[ia] : zero, ib >= 0 ? mass[ib] : zero, sA, sB, W.cMix[2 * cid],
				 W.cMix[2 * cid + 1], ( ia < 0 || ib < 0 ) ? sc.staticSoft : sc.contactSoft, sc.enableWarmStarting ? 1.0f : 0.0f );
	store_row_smem( m, local, cid, r );
	return make_int2( ia, ib );
}

/* Impulses of local row k back to its manifold (reference src/contact_solver.c:442-471,
 * :1180-1293): colour rows write both point slots, overflow rows their points. */
__device__ __forceinline__ void res_store( const b2gDevWorld& W, const SmemRows& m, int k, bool overflow )
{
	int4 idx = m.idx[k];
	b2gManifold* mf = W.manifold + idx.z;
	int n = overflow ? idx.w : 2;
	float4 imp[2] = { m.imp0[k], m.imp1[k] };
	float4 coef[2] = { m.coef0[k], m.coef1[k] };
#pragma unroll
	for ( int j = 0; j < 2; ++j )
	{
		if ( j >= n )
			break;
		mf->pts[j].normalImpulse = imp[j].x;
		mf->pts[j].tangentImpulse = imp[j].y;
		mf->pts[j].maxNormalImpulse = imp[j].z;
		mf->pts[j].normalVelocity = coef[j].w;
	}
}

__device__ __forceinline__ void res_terms( const b2gDevWorld& W, const ResBodies& rb, int k, int b, const b2gStepConst& sc )
{
	VelocityTerms v = velocity_terms( ( (const float4*)W.mass )[b], ( (const float4*)W.force )[b], ( (const float4*)W.extent )[b], sc );
	rb.term[k] = make_float4( v.lvd.x, v.lvd.y, v.avd, v.ld );
	rb.ad[k] = v.ad;
}

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
	for ( int k = tid, c = 0; k < rows; k += T )
	{
		while ( k >= share[c].base + share[c].count )
			++c;
		int2 e = res_prepare( W, m, share[c].first + ( k - share[c].base ), k, sc );
		top = max( top, max( e.x, e.y ) );
	}
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
	ResOverflow ov = res_carve_overflow( smem + P.ovOffset, P.ovOffset ? cs[B2G_COLORS] - cs[B2G_OVERFLOW] : 0 );
	if ( CL > 1 && rank == 0 && P.ovOffset )
	{
		res_index_overflow<T>( ov, m, share[B2G_OVERFLOW].base, cs[B2G_COLORS] - cs[B2G_OVERFLOW], &s_ovSlots );
		__syncthreads();
	}
	const int ids = top + 1;
	const int block = ids > 0 ? ( ids + CL - 1 ) / CL : 1;
	/* owners by a multiply-high with ceil(2^32 / block): exact for ids below 2^16 */
	if ( block <= P.bodyCap && ids < 65536 )
	{
		const unsigned inv = block > 1 ? (unsigned)( ( ( 1ull << 32 ) + (unsigned)block - 1 ) / (unsigned)block ) : 0u;
		DsmemBodies D{ { cl, rb.st0, rb.st1, block, rank, inv } };
		auto place = [&]( int b, int& r, int& s ) {
			r = CL == 1 ? 0 : ( block == 1 ? b : (int)__umulhi( (unsigned)b, inv ) );
			s = b - r * block;
		};
		auto there = [&]( int* p, int r ) { return CL == 1 ? p : cl.map_shared_rank( p, r ); };
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
		const int owned = min( block, ids - rank * block );
		for ( int s = tid; s < owned; s += T )
		{
			int b = rank * block + s;
			rb.st0[s] = gst[2 * b];
			rb.st1[s] = gst[2 * b + 1];
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
			res_run<CL, T, true>( P, share, m, LB, rb, gst, nullptr, awake, bar, rank, sc, ov, s_ovSlots );
		}
		else
			res_run<CL, T, true>( P, share, m, D, rb, gst, nullptr, awake, bar, rank, sc, ov, s_ovSlots );
		for ( int s = tid; s < owned; s += T )
		{
			int b = rank * block + s;
			int f = rb.flags[s];
			if ( f )
				gst[2 * b] = rb.st0[s];
			if ( f & RES_AWAKE )
				gst[2 * b + 1] = rb.st1[s];
		}
	}
	else
	{
		/* states at L2; the terms of this CTA's share of the list as far as they fit */
		L2Bodies G{ gst };
		const int n = al - af;
		if ( n <= P.bodyCap )
		{
			for ( int j = tid; j < n; j += T )
				res_terms( W, rb, j, W.awake[af + j], sc );
			bar.sync();
			res_run<CL, T, false>( P, share, m, G, rb, gst, W.awake + af, n, bar, rank, sc, ov, s_ovSlots );
		}
	}
	for ( int k = tid; k < rows; k += T )
		res_store( W, m, k, k >= colourRows );
}

/* The solver stage over a cooperative grid: body states in global memory, rows in shared
 * memory (ONCHIP) or in the row arrays, where row k of the colour-major order is entry k.
 * ctl: the barrier's arrival count, the count of finished CTAs and the give-up flag, all
 * zero at the launch and again when the kernel ends. */
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
	for ( int c = 0; c < B2G_COLORS; ++c )
		for ( int j = tid; j < share[c].count; j += T )
			res_prepare( W, m, share[c].first + j, share[c].base + j, sc );
	ResBodies rb;
	rb.st0 = rb.st1 = nullptr;
	rb.flags = rb.awake = nullptr;
	rb.term = smem + 9 * P.rowCap;
	rb.ad = (float*)( rb.term + P.bodyCap );
	const int af = res_first( P.awakeCount, rank, ctas );
	const int n = res_first( P.awakeCount, rank + 1, ctas ) - af;
	for ( int j = tid; j < n; j += T )
		res_terms( W, rb, j, W.awake[af + j], sc );
	ResOverflow ov = res_carve_overflow( smem + P.ovOffset, P.ovOffset ? ovRows : 0 );
	if ( rank == 0 && P.ovOffset )
	{
		__syncthreads();
		res_index_overflow<T>( ov, m, share[B2G_OVERFLOW].base, ovRows, &s_ovSlots );
	}
	ResBarrier<0> bar{ ctl, ctas, 0u };
	bar.sync();
	L2Bodies G{ (float4*)W.state };
	res_run<0, T, false>( P, share, m, G, rb, (float4*)W.state, W.awake + af, n, bar, rank, sc, ov, s_ovSlots );
	for ( int c = 0; c < B2G_COLORS; ++c )
		for ( int j = tid; j < share[c].count; j += T )
			res_store( W, m, share[c].base + j, c == B2G_OVERFLOW );
	if ( tid == 0 && atomicAdd( ctl + 1, 1 ) == ctas - 1 )
	{
		/* every CTA is past its last barrier */
		ctl[0] = 0;
		ctl[1] = 0;
		ctl[2] = 0;
	}
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

/* Row slots of the fullest CTA: every colour splits into shares that differ by one, CTA
 * 0 also holds the overflow rows. */
static int res_row_cap( const int* cs, int ctas )
{
	int cap = cs[B2G_COLORS] - cs[B2G_OVERFLOW];
	for ( int c = 0; c < B2G_OVERFLOW; ++c )
		cap += ( cs[c + 1] - cs[c] + ctas - 1 ) / ctas;
	return cap > 0 ? cap : 1;
}

/* Shared memory of CTA 0 with its overflow cache, which is left out when it does not fit. */
static size_t res_with_overflow( ResidentPlan* P, size_t bytes, int ovRows )
{
	P->ovOffset = 0;
	size_t at = ( bytes + 15 ) / 16;
	if ( ovRows > 0 && ovRows <= RES_OVERFLOW_MAX && 16 * at + res_overflow_bytes( ovRows ) <= RES_SMEM_MAX )
	{
		P->ovOffset = (int)at;
		bytes = 16 * at + res_overflow_bytes( ovRows );
	}
	return bytes;
}

/* The solver stage of caller buffers in one launch: the number of launches, 0 when this
 * device or set needs the per-phase kernels, or -1 on a launch error.  ctl: four ints of
 * device memory, zero, or cleared here when `clear` is set. */
extern "C" int b2gd_contact_resident( b2gDevWorld* w, const b2gSolvePlan* plan, const b2gStepConst* sc, int* ctl, int clear )
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

	/* One CTA, else a whole cluster, when the rows fit with as many bodies as the list
	 * has and one for every two rows (body indices are the caller's: the kernel copes
	 * with more, at L2).  One CTA is the faster one as long as it holds the set (1200
	 * contacts: 58 us, 80 in a cluster); clusters of 2, 4 or 8 take what 16 take (2000
	 * contacts: 78 to 82 us), so there is no space between the two; a grid is slower
	 * wherever a cluster holds the set (20000 contacts: 201 us, 110 in a cluster). */
	const int spaces[] = { 1, B2G_FUSED_CTAS };
	for ( int ctas : spaces )
	{
		if ( ctas > 1 && d->cluster == 0 )
			break;
		P.ctas = ctas;
		P.rowCap = res_row_cap( cs, ctas );
		int want = P.awakeCount > cs[B2G_COLORS] / 2 ? P.awakeCount : cs[B2G_COLORS] / 2;
		want = ( want + ctas - 1 ) / ctas + 1;
		size_t rows = 144u * (size_t)P.rowCap;
		size_t tail = ctas > 1 && ovRows > 0 && ovRows <= RES_OVERFLOW_MAX ? res_overflow_bytes( ovRows ) + 16 : 0;
		if ( rows + RES_BODY_BYTES * (size_t)want + tail > RES_SMEM_MAX )
			continue;
		/* the body slots take what the rows leave */
		P.bodyCap = (int)( ( RES_SMEM_MAX - rows - tail ) / RES_BODY_BYTES ) & ~3;
		if ( P.bodyCap > 4 * want )
			P.bodyCap = ( 4 * want + 3 ) & ~3;
		size_t bytes = rows + RES_BODY_BYTES * (size_t)P.bodyCap;
		if ( tail )
			bytes = res_with_overflow( &P, bytes, ovRows );
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
	P.ctas = ctas;
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
	if ( clear && cudaMemsetAsync( ctl, 0, 4 * sizeof( int ), s ) != cudaSuccess )
		return -1;
	size_t bytes = res_with_overflow( &P, 144u * (size_t)P.rowCap + terms, ovRows );
	auto kernel = onChip ? (ResGridKernel)k_solve_grid<GRID_THREADS, true> : (ResGridKernel)k_solve_grid<GRID_THREADS, false>;
	cudaLaunchConfig_t cfg = res_config( attr, ctas, 0, GRID_THREADS, bytes, s );
	return cudaLaunchKernelEx( &cfg, kernel, *w, P, *sc, ctl ) == cudaSuccess ? 1 : -1;
}
