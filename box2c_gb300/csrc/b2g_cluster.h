/*
 * b2g_cluster.h -- solver rows in shared memory and body states spread over the CTAs of
 * a thread-block cluster; shared by the fused single-world solver (fused.cu) and the
 * batched solver (batch.cu, rows of a world that fits in one CTA's shared memory).
 *
 * Rows use nine float4 arrays (structure of arrays): indices, normal / friction /
 * restitution, inverse masses, two anchor pairs, two coefficient sets, two impulse
 * sets; the softness follows from whether a body is static.  Body b lives in CTA
 * b / slots at slot b % slots; a body of the calling CTA is read and written in local
 * shared memory, any other through distributed shared memory.
 */
#pragma once

#include "b2g_solve.h"

#include <cooperative_groups.h>

namespace cg = cooperative_groups;

enum
{
	F_WARM = 0,
	F_SOLVE = 1,
	F_RELAX = 2,
	F_RESTITUTION = 3,
};

struct SmemRows
{
	int4* idx;	   /* ia ib contactId count */
	float4* nf;	   /* n.x n.y friction restitution */
	float4* ms;	   /* mA iA mB iB */
	float4* anc0;  /* rA.x rA.y rB.x rB.y of point 0 */
	float4* anc1;  /* point 1 */
	float4* coef0; /* base normalMass tangentMass relativeVelocity */
	float4* coef1;
	float4* imp0; /* normalImpulse tangentImpulse maxNormalImpulse 0 */
	float4* imp1;
};

/* Body states of the cluster: body b lives in CTA b / slots at slot b % slots.  A body
 * of this CTA is read and written in local shared memory, any other through
 * distributed shared memory. */
struct ClusterBodies
{
	cg::cluster_group cl;
	float4* st0;
	float4* st1;
	int slots;
	int rank;
	unsigned slotsInv; /* ceil(2^32 / slots) for slots > 1: b / slots = umulhi(b, slotsInv) for b, slots < 2^16 */

	__device__ __forceinline__ float4* word( float4* base, int b ) const
	{
		int r = slots == 1 ? b : (int)__umulhi( (unsigned)b, slotsInv );
		int s = b - r * slots;
		return r == rank ? base + s : cl.map_shared_rank( base + s, (unsigned)r );
	}

	/* full state (solve, relax, joints) */
	__device__ __forceinline__ DevState load( int b ) const
	{
		if ( b < 0 )
			return identity_state();
		return state_of( *word( st0, b ), *word( st1, b ) );
	}

	/* velocity only (warm start, restitution): dp and dq are not read */
	__device__ __forceinline__ DevState load_velocity( int b ) const
	{
		if ( b < 0 )
			return identity_state();
		return state_of( *word( st0, b ), make_float4( 0.0f, 0.0f, 1.0f, 0.0f ) );
	}

	__device__ __forceinline__ void store( int b, const DevState& x ) const
	{
		if ( b < 0 )
			return;
		*word( st0, b ) = velocity_word( x );
	}
};

__device__ __forceinline__ void load_row_smem( const SmemRows& m, int k, const b2gStepConst& sc, Row& r )
{
	int4 idx = m.idx[k];
	float4 nf = m.nf[k];
	float4 ms = m.ms[k];
	r.ia = idx.x;
	r.ib = idx.y;
	r.count = idx.w;
	r.n = gv( nf.x, nf.y );
	r.friction = nf.z;
	r.restitution = nf.w;
	const float* soft = ( idx.x < 0 || idx.y < 0 ) ? sc.staticSoft : sc.contactSoft;
	r.biasRate = soft[0];
	r.massScale = soft[1];
	r.impulseScale = soft[2];
	r.mA = ms.x;
	r.iA = ms.y;
	r.mB = ms.z;
	r.iB = ms.w;
	float4 a0 = m.anc0[k], a1 = m.anc1[k], c0 = m.coef0[k], c1 = m.coef1[k], i0 = m.imp0[k], i1 = m.imp1[k];
	r.rA[0] = gv( a0.x, a0.y );
	r.rB[0] = gv( a0.z, a0.w );
	r.rA[1] = gv( a1.x, a1.y );
	r.rB[1] = gv( a1.z, a1.w );
	r.base[0] = c0.x;
	r.nMass[0] = c0.y;
	r.tMass[0] = c0.z;
	r.relVel[0] = c0.w;
	r.base[1] = c1.x;
	r.nMass[1] = c1.y;
	r.tMass[1] = c1.z;
	r.relVel[1] = c1.w;
	r.ni[0] = i0.x;
	r.ti[0] = i0.y;
	r.maxNi[0] = i0.z;
	r.ni[1] = i1.x;
	r.ti[1] = i1.y;
	r.maxNi[1] = i1.z;
}

__device__ __forceinline__ void store_row_smem( const SmemRows& m, int k, int cid, const Row& r )
{
	m.idx[k] = make_int4( r.ia, r.ib, cid, r.count );
	m.nf[k] = make_float4( r.n.x, r.n.y, r.friction, r.restitution );
	m.ms[k] = make_float4( r.mA, r.iA, r.mB, r.iB );
	m.anc0[k] = make_float4( r.rA[0].x, r.rA[0].y, r.rB[0].x, r.rB[0].y );
	m.anc1[k] = make_float4( r.rA[1].x, r.rA[1].y, r.rB[1].x, r.rB[1].y );
	m.coef0[k] = make_float4( r.base[0], r.nMass[0], r.tMass[0], r.relVel[0] );
	m.coef1[k] = make_float4( r.base[1], r.nMass[1], r.tMass[1], r.relVel[1] );
	m.imp0[k] = make_float4( r.ni[0], r.ti[0], r.maxNi[0], 0.0f );
	m.imp1[k] = make_float4( r.ni[1], r.ti[1], r.maxNi[1], 0.0f );
}

/* Words of a manifold that a row's preparation reads: both points' anchors, separation,
 * normal and tangent impulse; the normal; the count. */
#define ROW_INPUTS 17
static_assert( sizeof( b2gPoint ) == 48 && sizeof( b2gManifold ) == 108, "manifold words" );

__device__ __forceinline__ void copy4_async( void* to, const void* from )
{
	asm volatile( "cp.async.ca.shared.global [%0], [%1], 4;" ::"r"( (unsigned)__cvta_generic_to_shared( to ) ), "l"( from ) );
}

__device__ __forceinline__ void copy16_async( void* to, const void* from )
{
	asm volatile( "cp.async.cg.shared.global [%0], [%1], 16;" ::"r"( (unsigned)__cvta_generic_to_shared( to ) ), "l"( from ) );
}

/* Preparation of rows [0, rows) in shared memory by T threads, whole warps (reference
 * src/contact_solver.c:597-808, :21-147): row k is entry source( k ) of the list (null: that
 * contact); source is called with growing k.  slot, when given, renumbers the bodies.
 *
 * Bound by latency: index, contact, bodies and manifold, row by row, is three round trips
 * to L2 for every T rows.  So a warp first fetches the indices of all its rows, then
 * starts the copies of all their inputs into the rows' own slots, and computes the rows
 * when they are there: three round trips in all.  Manifolds are 108 bytes apart; the warp
 * copies them as one stream of words, lane after lane.  What is left is the issue of the
 * copies (1130 rows in one CTA 10.4 -> 8.7 us, 1035 rows of a cluster's CTA 9.4 -> 7.7). */
template <class Source>
__device__ __forceinline__ void prepare_rows( const b2gDevWorld& W, const SmemRows& m, int rows, const int* list, const int* slot, Source source,
											  int thread, int T, const b2gStepConst& sc )
{
	constexpr int U = 4;
	for ( int k0 = thread; k0 < rows; k0 += U * T )
	{
		int cid[U], ia[U], ib[U];
#pragma unroll
		for ( int u = 0; u < U; ++u )
		{
			const int k = k0 + u * T;
			cid[u] = k < rows ? source( k ) : -1;
			if ( list && cid[u] >= 0 )
				cid[u] = list[cid[u]];
		}
#pragma unroll
		for ( int u = 0; u < U; ++u )
		{
			ia[u] = cid[u] >= 0 ? W.cBodies[2 * cid[u]] : -1;
			ib[u] = cid[u] >= 0 ? W.cBodies[2 * cid[u] + 1] : -1;
		}
#pragma unroll
		for ( int u = 0; u < U; ++u )
			if ( cid[u] >= 0 )
				m.idx[k0 + u * T] = make_int4( ia[u], ib[u], cid[u], 0 );
	}
	__syncwarp();
	const float4* gst = (const float4*)W.state;
	const float4* mass = (const float4*)W.mass;
	const int* words = (const int*)W.manifold;
	const int lane = thread & 31;
	const float4 zero = make_float4( 0.0f, 0.0f, 0.0f, 0.0f );
	const int stride = (int)( m.coef1 - m.coef0 );
	for ( int k0 = thread - lane; k0 < rows; k0 += T )
	{
		const int n = min( 32, rows - k0 );
		const int k = k0 + lane;
		const int4 own = lane < n ? m.idx[k] : make_int4( -1, -1, 0, 0 );
#pragma unroll
		for ( int i = 0; i < ROW_INPUTS; ++i )
		{
			const int t = lane + 32 * i, r = t / ROW_INPUTS, j = t - ROW_INPUTS * r;
			const int w = j < 7 ? j + 2 : ( j < 14 ? j + 7 : j + 10 );
			int* to = j < 16 ? (int*)( m.coef0 + ( j >> 2 ) * stride + k0 + r ) + ( j & 3 ) : &m.idx[k0 + r].w;
			const int c = __shfl_sync( 0xffffffffu, own.z, r );
			if ( r < n )
				copy4_async( to, words + 27 * (size_t)c + w );
		}
		if ( lane < n )
		{
			const int ia = own.x, ib = own.y, cid = own.z;
			copy4_async( &m.nf[k].z, W.cMix + 2 * cid );
			copy4_async( &m.nf[k].w, W.cMix + 2 * cid + 1 );
			if ( ia >= 0 )
			{
				copy16_async( m.anc0 + k, gst + 2 * ia );
				copy4_async( &m.ms[k].x, &mass[ia].y );
				copy4_async( &m.ms[k].y, &mass[ia].w );
				if ( slot != nullptr )
					copy4_async( &m.idx[k].x, slot + ia );
			}
			else
			{
				m.anc0[k] = zero;
				m.ms[k].x = m.ms[k].y = 0.0f;
			}
			if ( ib >= 0 )
			{
				copy16_async( m.anc1 + k, gst + 2 * ib );
				copy4_async( &m.ms[k].z, &mass[ib].y );
				copy4_async( &m.ms[k].w, &mass[ib].w );
				if ( slot != nullptr )
					copy4_async( &m.idx[k].y, slot + ib );
			}
			else
			{
				m.anc1[k] = zero;
				m.ms[k].z = m.ms[k].w = 0.0f;
			}
		}
	}
	asm volatile( "cp.async.wait_all;" ::: "memory" );
	__syncwarp();
	for ( int k = thread; k < rows; k += T )
	{
		const int4 ix = m.idx[k];
		const float4 nf = m.nf[k], ms = m.ms[k], a = m.anc0[k], b = m.anc1[k];
		const float4 q0 = m.coef0[k], q1 = m.coef1[k], q2 = m.imp0[k], q3 = m.imp1[k];
		b2gManifold in;
		in.pts[0].anchorA = gv( q0.x, q0.y );
		in.pts[0].anchorB = gv( q0.z, q0.w );
		in.pts[0].separation = q1.x;
		in.pts[0].normalImpulse = q1.y;
		in.pts[0].tangentImpulse = q1.z;
		in.pts[1].anchorA = gv( q1.w, q2.x );
		in.pts[1].anchorB = gv( q2.y, q2.z );
		in.pts[1].separation = q2.w;
		in.pts[1].normalImpulse = q3.x;
		in.pts[1].tangentImpulse = q3.y;
		in.normal = gv( q3.z, q3.w );
		in.count = ix.w;
		DevState sA = state_of( a, zero ), sB = state_of( b, zero );
		Row r;
		prepare_row( r, &in, ix.x, ix.y, make_float4( 0.0f, ms.x, 0.0f, ms.y ), make_float4( 0.0f, ms.z, 0.0f, ms.w ), sA, sB, nf.z, nf.w,
					 ( ix.x < 0 || ix.y < 0 ) ? sc.staticSoft : sc.contactSoft, sc.enableWarmStarting ? 1.0f : 0.0f );
		store_row_smem( m, k, ix.z, r );
	}
}

/* Impulses of rows [0, rows) back to their manifolds (reference src/contact_solver.c:442-471,
 * :1180-1293) by T threads: colour rows write both point slots, overflow rows
 * (from colourRows on) their points.  Eight threads a row, a word each, so that a
 * point's four words go out together: 1130 rows of one CTA 6.2 -> 1.7 us, 1035 rows of a
 * cluster's CTA 5.0 -> 1.6 us. */
__device__ __forceinline__ void store_impulses( const b2gDevWorld& W, const SmemRows& m, int rows, int colourRows, int thread, int T )
{
	float* words = (float*)W.manifold;
	for ( int t = thread; t < 8 * rows; t += T )
	{
		const int k = t >> 3, p = ( t >> 2 ) & 1, q = t & 3;
		const int4 idx = m.idx[k];
		if ( k >= colourRows && p >= idx.w )
			continue;
		const float4* from = q < 3 ? ( p ? m.imp1 : m.imp0 ) : ( p ? m.coef1 : m.coef0 );
		words[27 * (size_t)idx.z + 12 * p + 7 + q] = ( (const float*)( from + k ) )[q];
	}
}

/* One row phase on a row in shared memory; Bodies is ClusterBodies (states spread over
 * the cluster) or SharedBodies (states of one CTA, by body id). */
template <class Bodies>
__device__ __forceinline__ void row_step( const SmemRows& m, const Bodies& B, int k, int phase, bool scalar, const b2gStepConst& sc )
{
	Row r;
	load_row_smem( m, k, sc, r );
	bool delta = phase == F_SOLVE || phase == F_RELAX;
	DevState a = delta ? B.load( r.ia ) : B.load_velocity( r.ia );
	DevState b = delta ? B.load( r.ib ) : B.load_velocity( r.ib );
	bool changed = true;
	if ( phase == F_WARM )
		scalar ? warm_scalar( r, a, b ) : warm_lane( r, a, b );
	else if ( phase == F_SOLVE || phase == F_RELAX )
		scalar ? solve_scalar( r, a, b, phase == F_SOLVE, sc.inv_h, sc.pushout )
			   : solve_lane( r, a, b, phase == F_SOLVE, sc.inv_h, sc.pushout );
	else if ( scalar )
		changed = restitution_scalar( r, a, b, sc.restitutionThreshold );
	else
		restitution_lane( r, a, b, sc.restitutionThreshold );
	if ( changed == false )
		return;
	B.store( r.ia, a );
	B.store( r.ib, b );
	if ( phase != F_WARM )
	{
		m.imp0[k] = make_float4( r.ni[0], r.ti[0], r.maxNi[0], 0.0f );
		m.imp1[k] = make_float4( r.ni[1], r.ti[1], r.maxNi[1], 0.0f );
	}
}
