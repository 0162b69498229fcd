/*
 * b2g_push.h -- the solver stage over a cluster without cluster barriers: every CTA holds
 * copies of all bodies its rows touch, and an update goes to the other copies as an
 * asynchronous remote store that completes on the receiver's mbarrier.
 *
 * A sweep that reads and writes other CTAs' bodies in place costs a round trip to load
 * them, a store that has to be acknowledged before the barrier's release, and the
 * barrier.  Here a sweep reads only local shared memory, and waits for what other CTAs
 * send it in that sweep: one way, and not at all when nothing comes.  Large pyramid (16 CTAs,
 * 14950 rows): a sweep 0.88 -> 0.66 us, of which a wait for another CTA 0.17, the
 * exchange of the copies 5 us a step, the solver kernel 112 -> 97 us; tumbler of 2000
 * 370 -> 350 us.
 *
 * Who sends what is known before the first substep.  A body lives in the CTA that owns
 * its block of ids and has a copy in every CTA with a row or joint on it; each copy lists
 * the others (a mask of CTAs and its slot in each).  In one sweep at most one row of the
 * cluster moves a body (src/constraint_graph.c:84-131), so the bytes a CTA receives in a
 * sweep are 16 times the bodies of its copies that another CTA's rows of that colour
 * move: counted once, expected every time.
 *
 * One mbarrier per sweep of a substep, its phase the substep's parity.  A CTA cannot be
 * a substep ahead of one it shares a body with: each waits for the other's update of
 * that body (the owner for the row's, the row for the owner's integration) in every
 * substep.  So no arrival is counted into a phase before its own.
 */
#pragma once

#include "b2g_resident.h"

#define PUSH_CTAS B2G_FUSED_CTAS
/* mbarriers of a substep: velocity integration, four phases of an overflow sweep and up
 * to 12 colours, position integration */
#define PUSH_PHASE_BARS ( 1 + B2G_COLORS )
#define PUSH_BARS ( 2 + 4 * PUSH_PHASE_BARS )
#define PUSH_BAR_POSITION ( PUSH_BARS - 1 )
/* a CTA gives up on an mbarrier after this many polls or nanoseconds */
#define PUSH_SPIN_LIMIT ( 1 << 22 )
#define PUSH_SPIN_NS 1000000000ull
/* bytes of a copy: two state float4, its slots in the 16 CTAs, the mask of the others; of
 * an owned body besides: velocity terms, flags, an entry of the awake list */
#define PUSH_COPY_BYTES ( 32 + 2 * PUSH_CTAS + 4 )
#define PUSH_OWNED_BYTES ( 16 + 4 + 4 + 4 )
#define PUSH_LISTED 0x10000u /* in a mask: the copy is on the overflow list */

struct PushShared
{
	unsigned long long bar[PUSH_BARS];
	int colorBytes[B2G_COLORS]; /* received in a sweep of the active colour */
	int restBytes[B2G_COLORS];	/* in its restitution sweep */
	int ovBytes;				/* in an overflow sweep */
	int place[B2G_COLORS];		/* active index of a colour */
	int copies, fail, failAll, gaveUp, ovCount;
	int forwards; /* owned bodies that are sent but not integrated */
};

struct PushBodies : SharedBodies
{
	unsigned short* slot; /* PUSH_CTAS per copy */
	unsigned* mask;
	unsigned st0At, st1At, barAt; /* shared addresses; barAt of this sweep's mbarrier */

	__device__ __forceinline__ void send( unsigned base, int b, float4 v ) const
	{
		unsigned m = mask[b] & 0xffffu;
		while ( m != 0 )
		{
			const int t = __ffs( m ) - 1;
			m &= m - 1;
			unsigned to, bar;
			asm( "mapa.shared::cluster.u32 %0, %1, %2;" : "=r"( to ) : "r"( base + 16u * slot[PUSH_CTAS * b + t] ), "r"( t ) );
			asm( "mapa.shared::cluster.u32 %0, %1, %2;" : "=r"( bar ) : "r"( barAt ), "r"( t ) );
			asm volatile( "st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"( to ), "f"( v.x ),
						  "f"( v.y ), "f"( v.z ), "f"( v.w ), "r"( bar )
						  : "memory" );
		}
	}

	__device__ __forceinline__ void store( int b, const DevState& x ) const
	{
		if ( b < 0 )
			return;
		const float4 v = velocity_word( x );
		st0[b] = v;
		send( st0At, b, v );
	}
};

/* Begins sweep `bar`: the bytes it receives. */
__device__ __forceinline__ void push_expect( PushBodies& B, unsigned bars, int bar, int bytes )
{
	B.barAt = bars + 8u * (unsigned)bar;
	if ( threadIdx.x == 0 && bytes > 0 )
		asm volatile( "mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"( B.barAt ), "r"( bytes ) : "memory" );
}

/* Ends it: this CTA's own updates, then the ones it receives. */
__device__ __forceinline__ void push_wait( const PushBodies& B, PushShared& S, int bytes, int parity )
{
	__syncthreads();
	if ( bytes == 0 )
		return;
	unsigned long long start = 0;
	for ( int left = PUSH_SPIN_LIMIT;; )
	{
		unsigned done;
		asm volatile( "{ .reg .pred p; mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
					  : "=r"( done )
					  : "r"( B.barAt ), "r"( parity )
					  : "memory" );
		if ( done )
			return;
		bool late = --left == 0 || *(volatile int*)&S.gaveUp != 0;
		if ( ( left & 255 ) == 0 )
		{
			unsigned long long now;
			asm volatile( "mov.u64 %0, %globaltimer;" : "=l"( now ) );
			start = start == 0 ? now : start;
			late = late || now - start > PUSH_SPIN_NS;
		}
		if ( late )
		{
			*(volatile int*)&S.gaveUp = 1;
			return;
		}
	}
}

template <int PHASE, int T, bool JOINTS>
__device__ __forceinline__ void push_stage( const ResidentPlan& P, const ResShare* share, const SmemRows& m, const ResJoints& J, PushBodies& B,
											PushShared& S, unsigned bars, int rank, int sub, const int* ovList, const b2gStepConst& sc )
{
	const int* cs = P.colorStart;
	const int base = 1 + PHASE * PUSH_PHASE_BARS;
	const int parity = PHASE == F_RESTITUTION ? 0 : sub & 1;
	const int R = cs[B2G_COLORS] - cs[B2G_OVERFLOW];
	const int jointsAll = JOINTS ? P.jointStart[B2G_COLORS] - P.jointStart[B2G_OVERFLOW] : 0;
	if ( PHASE == F_RESTITUTION ? R > 0 : R + jointsAll > 0 )
	{
		const int bytes = S.ovBytes;
		push_expect( B, bars, base, bytes );
		if ( rank == 0 )
		{
			const ResShare o = share[B2G_OVERFLOW];
			if ( threadIdx.x == 0 )
			{
				const SharedBodies L = B;
				if ( JOINTS && PHASE != F_RESTITUTION )
					for ( int i = 0; i < jointsAll; ++i )
					{
						b2gJointDev* j = J.at( o.jfirst, o.jbase, i );
						res_joint( j, L, j->indexA, j->indexB, PHASE, sc );
					}
				for ( int i = 0; i < R; ++i )
					row_step( m, L, o.base + i, PHASE, true, sc );
			}
			__syncthreads();
			for ( int k = threadIdx.x; k < S.ovCount; k += T )
				B.send( B.st0At, ovList[k], B.st0[ovList[k]] );
		}
		push_wait( B, S, bytes, parity );
	}
	if ( PHASE == F_WARM && sc.enableWarmStarting == 0 )
		return;
	for ( int a = 0; a < P.activeCount; ++a )
	{
		const int c = P.active[a];
		if ( PHASE == F_RESTITUTION && cs[c + 1] == cs[c] )
			continue;
		const ResShare s = share[c];
		const int bytes = PHASE == F_RESTITUTION ? S.restBytes[a] : S.colorBytes[a];
		push_expect( B, bars, base + 1 + a, bytes );
		for ( int j = threadIdx.x; j < s.count; j += T )
			row_step( m, B, s.base + j, PHASE, false, sc );
		if ( JOINTS && PHASE != F_RESTITUTION )
			for ( int i = threadIdx.x; i < s.jcount; i += T )
			{
				b2gJointDev* j = J.at( s.jfirst, s.jbase, i );
				res_joint( j, B, j->indexA, j->indexB, PHASE, sc );
			}
		push_wait( B, S, bytes, parity );
	}
}

/* All substeps; rb: the owned bodies' terms and awake slots, the forwarded ones behind the
 * awake ones.  others: this CTA's copies of other CTAs' bodies. */
template <int T, bool JOINTS>
__device__ __forceinline__ void push_run( const ResidentPlan& P, const ResShare* share, const SmemRows& m, const ResJoints& J, PushBodies& B,
										  PushShared& S, const ResBodies& rb, int awake, int others, int rank, const int* ovList, const b2gStepConst& sc )
{
	const unsigned bars = (unsigned)__cvta_generic_to_shared( S.bar );
	const int bytes = 16 * others, sent = awake + S.forwards;
	for ( int sub = 0; sub < sc.subSteps; ++sub )
	{
		push_expect( B, bars, 0, bytes );
		for ( int j = threadIdx.x; j < sent; j += T )
		{
			const int s = rb.awake[j];
			DevState x = state_of( B.st0[s], make_float4( 0.0f, 0.0f, 1.0f, 0.0f ) );
			if ( j < awake )
			{
				float4 t4 = rb.term[s];
				VelocityTerms t;
				t.lvd = gv( t4.x, t4.y );
				t.avd = t4.z;
				t.ld = t4.w;
				t.ad = rb.ad[s];
				integrate_velocity( x, t, sc );
			}
			B.store( s, x );
		}
		push_wait( B, S, bytes, sub & 1 );
		push_stage<F_WARM, T, JOINTS>( P, share, m, J, B, S, bars, rank, sub, ovList, sc );
		push_stage<F_SOLVE, T, JOINTS>( P, share, m, J, B, S, bars, rank, sub, ovList, sc );
		push_expect( B, bars, PUSH_BAR_POSITION, bytes );
		for ( int j = threadIdx.x; j < sent; j += T )
		{
			const int s = rb.awake[j];
			DevState x = state_of( B.st0[s], B.st1[s] );
			if ( j < awake )
				integrate_position( x, sc.h );
			const float4 v = make_float4( x.dp.x, x.dp.y, x.dq.c, x.dq.s );
			B.st1[s] = v;
			B.send( B.st1At, s, v );
		}
		push_wait( B, S, bytes, sub & 1 );
		push_stage<F_RELAX, T, JOINTS>( P, share, m, J, B, S, bars, rank, sub, ovList, sc );
	}
	push_stage<F_RESTITUTION, T, JOINTS>( P, share, m, J, B, S, bars, rank, 0, ovList, sc );
}

/* Carves copies after the rows: st0, st1, owned terms, slots, masks, owned ad / flags /
 * awake.  cap copies, of which the first `owned` are the CTA's own bodies. */
__device__ __forceinline__ void push_carve( float4* base, int cap, int owned, PushBodies& B, ResBodies& rb )
{
	B.st0 = base;
	B.st1 = base + cap;
	rb.st0 = B.st0;
	rb.st1 = B.st1;
	rb.term = base + 2 * cap;
	B.slot = (unsigned short*)( rb.term + owned );
	B.mask = (unsigned*)( B.slot + PUSH_CTAS * cap );
	rb.ad = (float*)( B.mask + cap );
	rb.flags = (int*)( rb.ad + owned );
	rb.awake = rb.flags + owned;
	B.st0At = (unsigned)__cvta_generic_to_shared( B.st0 );
	B.st1At = (unsigned)__cvta_generic_to_shared( B.st1 );
	B.barAt = 0;
}

/* Before the CTAs meet for the first time: barriers and counts of this CTA, and of its
 * owned copies the slot and an empty mask.  All threads. */
__device__ __forceinline__ void push_init( PushBodies& B, PushShared& S, const ResidentPlan& P, int owned, int rank )
{
	const int tid = threadIdx.x;
	if ( tid == 0 )
	{
		const unsigned bars = (unsigned)__cvta_generic_to_shared( S.bar );
		for ( int i = 0; i < PUSH_BARS; ++i )
			asm volatile( "mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"( bars + 8u * (unsigned)i ) : "memory" );
		asm volatile( "fence.mbarrier_init.release.cluster;" ::: "memory" );
		S.ovBytes = 0;
		S.copies = owned;
		S.fail = S.failAll = S.gaveUp = S.ovCount = S.forwards = 0;
		for ( int a = 0; a < P.activeCount; ++a )
			S.place[P.active[a]] = a;
	}
	if ( tid < B2G_COLORS )
		S.colorBytes[tid] = S.restBytes[tid] = 0;
	for ( int s = tid; s < owned; s += blockDim.x )
	{
		B.mask[s] = 0;
		B.slot[PUSH_CTAS * s + rank] = (unsigned short)s;
	}
}

/* A body end of a row or joint: the CTA gets a copy the first time it meets the body.
 * owner, at: where the body lives. */
__device__ __forceinline__ void push_meet( const cg::cluster_group& cl, const PushBodies& B, PushShared& S, int cap, int rank, int owner, int at )
{
	if ( owner == rank )
		return;
	const unsigned bit = 1u << rank;
	if ( atomicOr( cl.map_shared_rank( B.mask + at, owner ), bit ) & bit )
		return;
	const int s = atomicAdd( &S.copies, 1 );
	if ( s >= cap )
	{
		S.fail = 1;
		return;
	}
	*cl.map_shared_rank( B.slot + PUSH_CTAS * at + rank, owner ) = (unsigned short)s;
	/* the new copy's entry says where it comes from until it is filled */
	B.slot[PUSH_CTAS * s] = (unsigned short)owner;
	B.slot[PUSH_CTAS * s + 1] = (unsigned short)at;
}

/* Fills this CTA's copies of other CTAs' bodies. */
__device__ __forceinline__ void push_fill( const cg::cluster_group& cl, PushBodies& B, PushShared& S, int owned, int rank )
{
	for ( int s = owned + threadIdx.x; s < S.copies; s += blockDim.x )
	{
		const int owner = B.slot[PUSH_CTAS * s], at = B.slot[PUSH_CTAS * s + 1];
		B.st0[s] = *cl.map_shared_rank( B.st0 + at, owner );
		B.st1[s] = *cl.map_shared_rank( B.st1 + at, owner );
		const unsigned m = *cl.map_shared_rank( B.mask + at, owner );
		B.mask[s] = ( m | ( 1u << owner ) ) & ~( 1u << rank ) & 0xffffu;
		const uint4* from = cl.map_shared_rank( (const uint4*)( B.slot + PUSH_CTAS * at ), owner );
		uint4* to = (uint4*)( B.slot + PUSH_CTAS * s );
		const uint4 w0 = from[0], w1 = from[1];
		to[0] = w0;
		to[1] = w1;
	}
}

/* This CTA's copy of a body. */
__device__ __forceinline__ int push_slot( const cg::cluster_group& cl, const PushBodies& B, int rank, int owner, int at )
{
	return owner == rank ? at : (int)*cl.map_shared_rank( B.slot + PUSH_CTAS * at + rank, owner );
}

/* Tells the other copies' CTAs that a row (or joint) of colour c here moves copy s; of an
 * overflow constraint, that the overflow pass does. */
__device__ __forceinline__ void push_count( const cg::cluster_group& cl, const PushBodies& B, PushShared& S, int s, int c, bool row, int* ovList )
{
	if ( c == B2G_OVERFLOW )
	{
		if ( atomicOr( B.mask + s, PUSH_LISTED ) & PUSH_LISTED )
			return;
		ovList[atomicAdd( &S.ovCount, 1 )] = s;
	}
	unsigned m = B.mask[s] & 0xffffu;
	while ( m != 0 )
	{
		const int t = __ffs( m ) - 1;
		m &= m - 1;
		if ( c == B2G_OVERFLOW )
			atomicAdd( cl.map_shared_rank( &S.ovBytes, t ), 16 );
		else
		{
			atomicAdd( cl.map_shared_rank( S.colorBytes + S.place[c], t ), 16 );
			if ( row )
				atomicAdd( cl.map_shared_rank( S.restBytes + S.place[c], t ), 16 );
		}
	}
}

/* From rows and joints on body ids to rows and joints on copies, with the expected bytes
 * counted; false, on every CTA, when a CTA's copies do not fit: the ids are unchanged
 * then.  Owned bodies (of block ids a CTA, inv its reciprocal) are in the first slots of
 * their owners; behind the `awake` ones of rb.awake, which integrated( s ) knows, come the
 * others with copies elsewhere.  All threads of the cluster; the caller meets the other
 * CTAs before the first sweep. */
template <bool JOINTS, class F>
__device__ __forceinline__ bool push_exchange( const cg::cluster_group& cl, PushBodies& B, PushShared& S, int cap, int block, unsigned inv, int rank,
											   int rows, int joints, const ResShare* share, const SmemRows& m, const ResJoints& J, int* ovList,
											   const ResBodies& rb, const int& awake, F integrated )
{
	const int tid = threadIdx.x, T = blockDim.x;
	auto owner_of = [&]( int b ) { return block == 1 ? b : (int)__umulhi( (unsigned)b, inv ); };
	auto meet = [&]( int b ) {
		if ( b >= 0 )
			push_meet( cl, B, S, cap, rank, owner_of( b ), b - owner_of( b ) * block );
	};
	auto take = [&]( int b ) { return b < 0 ? -1 : push_slot( cl, B, rank, owner_of( b ), b - owner_of( b ) * block ); };
	auto tell = [&]( int s, int c, bool row ) {
		if ( s >= 0 )
			push_count( cl, B, S, s, c, row, ovList );
	};
	auto joint_at = [&]( int k, int& c ) {
		while ( k >= share[c].jbase + share[c].jcount )
			++c;
		return J.at( share[c].jfirst, share[c].jbase, k - share[c].jbase );
	};
	cl.sync();
	for ( int k = tid; k < rows; k += T )
	{
		meet( m.idx[k].x );
		meet( m.idx[k].y );
	}
	if ( JOINTS )
		for ( int k = tid, c = 0; k < joints; k += T )
		{
			const b2gJointDev* j = joint_at( k, c );
			meet( j->indexA );
			meet( j->indexB );
		}
	__syncthreads();
	if ( tid < PUSH_CTAS && S.fail )
		*cl.map_shared_rank( &S.failAll, tid ) = 1;
	cl.sync();
	if ( S.failAll )
		return false;
	push_fill( cl, B, S, block, rank );
	for ( int s = tid; s < block; s += T )
		if ( ( B.mask[s] & 0xffffu ) != 0 && integrated( s ) == false )
			rb.awake[awake + atomicAdd( &S.forwards, 1 )] = s;
	__syncthreads();
	for ( int k = tid, c = 0; k < rows; k += T )
	{
		while ( k >= share[c].base + share[c].count )
			++c;
		const int a = take( m.idx[k].x ), b = take( m.idx[k].y );
		m.idx[k].x = a;
		m.idx[k].y = b;
		tell( a, c, true );
		tell( b, c, true );
	}
	if ( JOINTS )
		for ( int k = tid, c = 0; k < joints; k += T )
		{
			b2gJointDev* j = joint_at( k, c );
			const int a = take( j->indexA ), b = take( j->indexB );
			j->indexA = a;
			j->indexB = b;
			tell( a, c, false );
			tell( b, c, false );
		}
	return true;
}
