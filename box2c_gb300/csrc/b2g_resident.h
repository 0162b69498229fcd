/*
 * b2g_resident.h -- the parts of a resident solver stage: constraint rows and joints held
 * on chip, the stages over them, barriers between sweeps, row preparation and impulse
 * storage.  resident.cu builds the kernels on caller buffers from them, fused.cu those of
 * a world's step.
 */
#pragma once

#include "b2g_cluster.h"
#include "b2g_device.h"
#include "b2g_space.h"
#include "b2g_stages.h"

#include <cuda_runtime.h>

/* polls of a grid barrier before it gives up (seconds; a cooperative launch never gets
 * there) */
#ifndef RES_SPIN_LIMIT
#define RES_SPIN_LIMIT ( 1 << 22 )
#endif

struct ResidentPlan
{
	int colorStart[B2G_COLORS + 1];
	int jointStart[B2G_COLORS + 1];
	int active[B2G_COLORS];
	int activeCount;
	int awakeCount;
	int bodyIdCount; /* body ids of a world (0: caller buffers, ids unknown) */
	int rowCap;	  /* row slots per CTA (0: rows in the row arrays) */
	int bodyCap;  /* body slots per CTA in shared memory; a grid's velocity-term slots */
	int jointCap; /* joint slots per CTA in shared memory (0: joints in the joint array) */
	int jointOffset; /* float4 offset of the joint slots */
	int bodyOffset;	 /* float4 offset of a cluster's body slots */
	int pushCap;	 /* body copies per CTA (0: no copies) */
	int pushBytes;	 /* caller buffers, whose copies the kernel counts: their shared memory */
	int ovOffset; /* float4 offset of the overflow cache, 0 without one */
};

/* Overflow cache of CTA 0: for R overflow rows and J overflow joints with E = 2 (R + J)
 * body ends, the rows' indices with body slots (int4 x R), slot states (2 x float4 x E),
 * slot bodies, first occurrences and slots per end (3 x int x E), joint slots (int2 x J). */
struct ResOverflow
{
	int4* idx;
	float4* st0;
	float4* st1;
	int* body;
	int* first;
	int* slot;
	int2* jslot;
};

__device__ __forceinline__ ResOverflow res_carve_overflow( float4* base, int R, int J )
{
	int E = 2 * ( R + J );
	ResOverflow o;
	o.idx = (int4*)base;
	o.st0 = base + R;
	o.st1 = o.st0 + E;
	o.body = (int*)( o.st1 + E );
	o.first = o.body + E;
	o.slot = o.first + E;
	o.jslot = (int2*)( o.slot + E );
	return o;
}

/* A joint's record in shared memory: 65 words apart, so that the threads of a warp, each
 * on its own joint, read different banks. */
#define RES_JOINT_WORDS ( (int)( sizeof( b2gJointDev ) / 4 ) + 1 )
#define RES_JOINT_BYTES ( 4 * RES_JOINT_WORDS )

struct ResBodies
{
	float4* st0;  /* v.x v.y w tag */
	float4* st1;  /* dp.x dp.y dq.c dq.s */
	float4* term; /* lvd.x lvd.y avd ld */
	float* ad;	  /* angular damping factor */
	int* flags;	  /* RES_AWAKE, RES_TOUCHED; of a world: awake indices */
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

/* One CTA's share of a colour: rows [first, first + count) of the colour-major order at
 * local index base, joints [jfirst, jfirst + jcount) of the joint list at jbase. */
struct ResShare
{
	int first, count, base;
	int jfirst, jcount, jbase;
};

/* Where the joints are: CTA-local records, or the world's joint array through the list. */
struct ResJoints
{
	char* local; /* null: in the joint array */
	b2gJointDev* array;
	const int* list;
	__device__ __forceinline__ b2gJointDev* at( int jfirst, int jbase, int i ) const
	{
		return local ? (b2gJointDev*)( local + (size_t)RES_JOINT_BYTES * (size_t)( jbase + i ) ) : array + list[jfirst + i];
	}
};

template <class Bodies>
__device__ __forceinline__ void res_joint( b2gJointDev* j, const Bodies& B, int ia, int ib, int phase, const b2gStepConst& sc )
{
	DevState a = B.load( ia );
	DevState b = B.load( ib );
	if ( phase == F_WARM )
		joint_warm_state( j, a, b );
	else
		joint_solve_state( j, a, b, phase == F_SOLVE, sc );
	B.store( ia, a );
	B.store( ib, b );
}

__device__ __forceinline__ int res_first( int n, int k, int ctas ) { return (int)( (long long)n * k / ctas ); }

/* One stage over all colours: the overflow set first (serially, CTA 0), then each active
 * colour with a barrier after it.  T threads a CTA (0: as launched).  PART:
 * the one CTA of a bin, which holds a part of the plan's rows and joints.  JOINTS false compiles the joints out. */
template <int CL, int PHASE, int T, bool JOINTS, bool PART, class Bodies>
__device__ __forceinline__ void res_stage( const ResidentPlan& P, const ResShare* share, const SmemRows& m, const ResJoints& J, const Bodies& B,
										   ResBarrier<CL>& bar, int rank, const b2gStepConst& sc, const ResOverflow& ov, int ovSlots )
{
	const int* cs = P.colorStart;
	const int R = PART ? share[B2G_OVERFLOW].count : cs[B2G_COLORS] - cs[B2G_OVERFLOW];
	const int jointsAll = JOINTS ? ( PART ? share[B2G_OVERFLOW].jcount : P.jointStart[B2G_COLORS] - P.jointStart[B2G_OVERFLOW] ) : 0;
	const int joints = PHASE == F_RESTITUTION ? 0 : jointsAll;
	const int step = T ? T : (int)blockDim.x;
	if ( PHASE == F_RESTITUTION ? R > 0 : R + jointsAll > 0 )
	{
		if ( rank == 0 )
		{
			const ResShare o = share[B2G_OVERFLOW];
			if ( CL != 1 && P.ovOffset != 0 )
			{
				/* the set's bodies to local slots, the serial pass on them, velocities back:
				 * nothing else touches a body while the set runs */
				for ( int s = threadIdx.x; s < ovSlots; s += step )
				{
					int b = ov.body[s];
					ov.st0[s] = B.word0( b );
					ov.st1[s] = B.word1( b );
				}
				__syncthreads();
				if ( threadIdx.x == 0 )
				{
					SharedBodies OB{ ov.st0, ov.st1 };
					if ( JOINTS )
						for ( int i = 0; i < joints; ++i )
							res_joint( J.at( o.jfirst, o.jbase, i ), OB, ov.jslot[i].x, ov.jslot[i].y, PHASE, sc );
					SmemRows mo = { ov.idx, m.nf + o.base, m.ms + o.base, m.anc0 + o.base, m.anc1 + o.base, m.coef0 + o.base, m.coef1 + o.base,
									m.imp0 + o.base, m.imp1 + o.base };
					for ( int i = 0; i < R; ++i )
						row_step( mo, OB, i, PHASE, true, sc );
				}
				__syncthreads();
				for ( int s = threadIdx.x; s < ovSlots; s += step )
					B.set_word0( ov.body[s], ov.st0[s] );
			}
			else if ( threadIdx.x == 0 )
			{
				if ( JOINTS )
					for ( int i = 0; i < joints; ++i )
					{
						b2gJointDev* j = J.at( o.jfirst, o.jbase, i );
						res_joint( j, B, j->indexA, j->indexB, PHASE, sc );
					}
				for ( int i = 0; i < R; ++i )
					row_step( m, B, o.base + i, PHASE, true, sc );
			}
		}
		bar.sync();
	}
	if ( PHASE == F_WARM && sc.enableWarmStarting == 0 )
		return;
	for ( int a = 0; a < P.activeCount; ++a )
	{
		const int c = P.active[a];
		if ( JOINTS && PHASE == F_RESTITUTION && cs[c + 1] == cs[c] )
			continue;
		const ResShare s = share[c];
		if ( PART && s.count + ( JOINTS && PHASE != F_RESTITUTION ? s.jcount : 0 ) == 0 )
			continue;
		for ( int j = threadIdx.x; j < s.count; j += step )
			row_step( m, B, s.base + j, PHASE, false, sc );
		if ( JOINTS && PHASE != F_RESTITUTION )
			for ( int i = threadIdx.x; i < s.jcount; i += step )
			{
				b2gJointDev* j = J.at( s.jfirst, s.jbase, i );
				res_joint( j, B, j->indexA, j->indexB, PHASE, sc );
			}
		bar.sync();
	}
}

/* All substeps over bodies B.  Integration runs over this CTA's awake bodies: with states
 * in shared memory slots b.awake[0 .. awake), in global memory the ids list[0 .. awake). */
template <int CL, int T, bool SHARED_STATES, bool JOINTS, bool PART = false, class Bodies>
__device__ __forceinline__ void res_run( const ResidentPlan& P, const ResShare* share, const SmemRows& m, const ResJoints& J, const Bodies& B,
										 const ResBodies& rb, float4* gst, const int* list, int awake, ResBarrier<CL>& bar, int rank,
										 const b2gStepConst& sc, const ResOverflow& ov, int ovSlots )
{
	const int step = T ? T : (int)blockDim.x;
	for ( int sub = 0; sub < sc.subSteps; ++sub )
	{
		for ( int j = threadIdx.x; j < awake; j += step )
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
		res_stage<CL, F_WARM, T, JOINTS, PART>( P, share, m, J, B, bar, rank, sc, ov, ovSlots );
		res_stage<CL, F_SOLVE, T, JOINTS, PART>( P, share, m, J, B, bar, rank, sc, ov, ovSlots );
		for ( int j = threadIdx.x; j < awake; j += step )
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
		res_stage<CL, F_RELAX, T, JOINTS, PART>( P, share, m, J, B, bar, rank, sc, ov, ovSlots );
	}
	res_stage<CL, F_RESTITUTION, T, JOINTS, PART>( P, share, m, J, B, bar, rank, sc, ov, ovSlots );
}

/* Overflow cache: the distinct bodies of the set's ends (joints first) get slots in end
 * order. */
template <int T, bool JOINTS>
__device__ __forceinline__ void res_index_overflow( const ResOverflow& ov, const SmemRows& m, const ResJoints& J, const ResShare& o, int joints,
													int R, int* slots )
{
	const int nj = JOINTS ? joints : 0;
	const int step = T ? T : (int)blockDim.x;
	const int E = 2 * ( R + nj );
	auto end_body = [&]( int e ) {
		if ( JOINTS && e < 2 * nj )
		{
			const b2gJointDev* j = J.at( o.jfirst, o.jbase, e >> 1 );
			return ( e & 1 ) ? j->indexB : j->indexA;
		}
		int4 ix = m.idx[o.base + ( ( e - 2 * nj ) >> 1 )];
		return ( e & 1 ) ? ix.y : ix.x;
	};
	for ( int e = threadIdx.x; e < E; e += step )
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
	for ( int e = threadIdx.x; e < E; e += step )
	{
		int f = ov.first[e];
		int s = f < 0 ? -1 : ov.slot[f];
		if ( JOINTS && e < 2 * nj )
		{
			if ( e & 1 )
				ov.jslot[e >> 1].y = s;
			else
				ov.jslot[e >> 1].x = s;
			continue;
		}
		int r = ( e - 2 * nj ) >> 1;
		if ( e & 1 )
			ov.idx[r].y = s;
		else
		{
			int4 ix = m.idx[o.base + r];
			ov.idx[r].x = s;
			ov.idx[r].z = ix.z;
			ov.idx[r].w = ix.w;
		}
	}
}

/* Preparation of one row in the row arrays: contact k. */
__device__ __forceinline__ void res_prepare_global( const b2gDevWorld& W, const SmemRows& m, int k, const b2gStepConst& sc )
{
	const float4* gst = (const float4*)W.state;
	const float4* mass = (const float4*)W.mass;
	const float4 zero = make_float4( 0.0f, 0.0f, 0.0f, 0.0f );
	int ia = W.cBodies[2 * k];
	int ib = W.cBodies[2 * k + 1];
	DevState sA = ia >= 0 ? state_of( gst[2 * ia], gst[2 * ia + 1] ) : identity_state();
	DevState sB = ib >= 0 ? state_of( gst[2 * ib], gst[2 * ib + 1] ) : identity_state();
	Row r;
	prepare_row( r, W.manifold + k, ia, ib, ia >= 0 ? mass[ia] : zero, ib >= 0 ? mass[ib] : zero, sA, sB, W.cMix[2 * k], W.cMix[2 * k + 1],
				 ( ia < 0 || ib < 0 ) ? sc.staticSoft : sc.contactSoft, sc.enableWarmStarting ? 1.0f : 0.0f );
	store_row_smem( m, k, k, r );
}

/* The list entry of local row k; k grows from call to call of one thread. */
struct ResSource
{
	const ResShare* share;
	int c;
	__device__ __forceinline__ int operator()( int k )
	{
		while ( k >= share[c].base + share[c].count )
			++c;
		return share[c].first + ( k - share[c].base );
	}
};

__device__ __forceinline__ void res_terms( const b2gDevWorld& W, const ResBodies& rb, int k, int b, const b2gStepConst& sc )
{
	VelocityTerms v = velocity_terms( ( (const float4*)W.mass )[b], ( (const float4*)W.force )[b], ( (const float4*)W.extent )[b], sc );
	rb.term[k] = make_float4( v.lvd.x, v.lvd.y, v.avd, v.ld );
	rb.ad[k] = v.ad;
}
