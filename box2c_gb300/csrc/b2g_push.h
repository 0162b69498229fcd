/*
 * b2g_push.h -- the solver stage over a cluster without cluster barriers: every CTA holds
 * copies of all bodies its rows touch, and an update goes to the other copies as an
 * asynchronous remote store that completes on the receiver's mbarrier.
 *
 * A sweep that reads and writes other CTAs' bodies in place costs a round trip to load
 * them, a store that has to be acknowledged before the barrier's release, and the
 * barrier.  Here a sweep reads only local shared memory, and waits for what other CTAs
 * send it in that sweep: one way, and not at all when nothing comes.  Large pyramid (16 CTAs,
 * 14950 rows): a sweep 0.88 -> 0.57 us, the exchange of the copies 8 us a step, the solver
 * stage 112 -> 94 us; tumbler of 2000 370 -> 337 us.
 *
 * Who sends what is known before the first substep.  A body lives in the CTA that owns
 * its block of ids and has a copy in every CTA with a row or joint on it.  In one sweep at
 * most one row of the cluster moves a body (src/constraint_graph.c:84-131), so its
 * velocity passes from one update to the next: the owner's integration, the rows of the
 * stage in the order of their colours, again for the next stage, the owner.  An update
 * sends the velocity to the one CTA that updates it next (b2g_chain.h), or keeps it; the
 * position, which only the owner updates, goes to all copies, and to the next updater the
 * velocity with it.  The bytes a CTA receives in a sweep are counted once and expected
 * every time.
 *
 * So no two writes of a copy are under way at once, though nothing orders remote stores
 * of different CTAs: a CTA is sent a velocity only to update it, and whoever sends it the
 * next one has, by way of the CTAs between, received that update.  The same holds for
 * the positions: every CTA with a copy updates the velocity between two of them.
 *
 * One mbarrier per sweep of a substep, its phase the substep's parity.  By the same chain
 * no bytes are counted into a phase before its own: an update that a CTA is sent in a
 * substep follows its own update, and so its wait, in the one before.  For that the owner
 * takes part with bodies that it does not integrate as well, unchanged.
 */
#pragma once

#include "b2g_chain.h"
#include "b2g_resident.h"

#define PUSH_CTAS B2G_FUSED_CTAS
/* mbarriers: velocity integration, four phases of up to 12 places, position integration,
 * the start of restitution */
#define PUSH_BARS ( 3 + 4 * B2G_CHAIN_PLACES )
#define PUSH_BAR_POSITION ( PUSH_BARS - 2 )
#define PUSH_BAR_RESTITUTION ( PUSH_BARS - 1 )
/* a CTA gives up on an mbarrier after this many polls or nanoseconds; then all of the
 * cluster leave the solve at the next substep, and its results are marked */
#ifndef PUSH_SPIN_LIMIT
#define PUSH_SPIN_LIMIT ( 1 << 22 )
#endif
#define PUSH_SPIN_NS 1000000000ull
/* what a store under way to another CTA may take: a cluster that gave up waits it out */
#define PUSH_FLIGHT_NS 100000ull
/* bytes of a copy: two state float4, its slots in the 16 CTAs, the mask of the others; of
 * an owned body besides: velocity terms, chain, damping, flags, an entry of the awake list */
#define PUSH_COPY_BYTES ( 32 + 2 * PUSH_CTAS + 4 )
#define PUSH_OWNED_BYTES ( 16 + 16 + 4 + 4 + 4 )
#define PUSH_LISTED 0x10000u /* in a mask: the copy is on the overflow list */
/* A body of a row or joint: its copy's slot in 16 bits, then the CTAs that need the
 * velocity after a warm start, a solve or relaxation, and a restitution, 4 bits each. */
#define PUSH_SLOT 0xffff
#define PUSH_NEXT( b, phase ) ( ( ( b ) >> ( ( phase ) == F_WARM ? 16 : ( phase ) == F_RESTITUTION ? 24 : 20 ) ) & 15 )

static_assert( B2G_CHAIN_PLACES == B2G_COLORS && PUSH_CTAS == 16, "places and CTAs of a chain" );

struct PushShared
{
	unsigned long long bar[PUSH_BARS];
	/* velocities received in a sweep of a place: in a warm start, and times 65536 in a
	 * solve or relaxation; in restitution */
	int moved[B2G_CHAIN_PLACES], rest[B2G_CHAIN_PLACES];
	int firsts, restFirsts; /* after an integration, at the start of restitution */
	int place[B2G_COLORS];	/* of a colour */
	int copies, fail, failAll, gaveUp, ovCount;
	int forwards; /* owned bodies that are sent but not integrated */
};

struct PushBodies : SharedBodies
{
	unsigned short* slot; /* PUSH_CTAS per copy */
	unsigned* mask;
	uint4* chain; /* of an owned body: who, cta; the CTAs that come first, in restitution 16 times */
	int rank;
	unsigned st0At, st1At, barAt; /* shared addresses; barAt of this sweep's mbarrier */

	__device__ __forceinline__ void send( unsigned base, int s, int t, float4 v ) const
	{
		unsigned to, bar;
		asm( "mapa.shared::cluster.u32 %0, %1, %2;" : "=r"( to ) : "r"( base + 16u * slot[PUSH_CTAS * s + t] ), "r"( t ) );
		asm( "mapa.shared::cluster.u32 %0, %1, %2;" : "=r"( bar ) : "r"( barAt ), "r"( t ) );
		asm volatile( "st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"( to ), "f"( v.x ),
					  "f"( v.y ), "f"( v.z ), "f"( v.w ), "r"( bar )
					  : "memory" );
	}
	/* to the next updater, which may be this CTA */
	__device__ __forceinline__ void pass( int s, int t, float4 v ) const
	{
		if ( t == rank )
			st0[s] = v;
		else
			send( st0At, s, t, v );
	}
	__device__ __forceinline__ void send_position( int s, float4 v ) const
	{
		unsigned m = mask[s] & 0xffffu;
		while ( m != 0 )
		{
			const int t = __ffs( m ) - 1;
			m &= m - 1;
			send( st1At, s, t, v );
		}
	}
};

/* The bodies of the rows and joints of a stage. */
template <int PHASE>
struct PushStage : PushBodies
{
	__device__ __forceinline__ DevState load( int b ) const
	{
		return b < 0 ? identity_state() : state_of( st0[b & PUSH_SLOT], st1[b & PUSH_SLOT] );
	}
	__device__ __forceinline__ DevState load_velocity( int b ) const
	{
		return b < 0 ? identity_state() : state_of( st0[b & PUSH_SLOT], make_float4( 0.0f, 0.0f, 1.0f, 0.0f ) );
	}
	__device__ __forceinline__ void store( int b, const DevState& x ) const
	{
		if ( b >= 0 )
			pass( b & PUSH_SLOT, PUSH_NEXT( b, PHASE ), velocity_word( x ) );
	}
};

/* The same in an overflow set, whose updates are passed on when it is done. */
struct PushOverflow : SharedBodies
{
	__device__ __forceinline__ DevState load( int b ) const { return SharedBodies::load( b < 0 ? b : b & PUSH_SLOT ); }
	__device__ __forceinline__ DevState load_velocity( int b ) const { return SharedBodies::load_velocity( b < 0 ? b : b & PUSH_SLOT ); }
	__device__ __forceinline__ void store( int b, const DevState& x ) const { SharedBodies::store( b < 0 ? b : b & PUSH_SLOT, x ); }
};

/* Begins sweep `bar`: the bytes it receives. */
__device__ __forceinline__ void push_expect( PushBodies& B, unsigned bars, int bar, int bytes )
{
	B.barAt = bars + 8u * (unsigned)bar;
	if ( threadIdx.x == 0 && bytes > 0 )
		asm volatile( "mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"( B.barAt ), "r"( bytes ) : "memory" );
}

__device__ __forceinline__ unsigned long long push_clock()
{
	unsigned long long now;
	asm volatile( "mov.u64 %0, %globaltimer;" : "=l"( now ) );
	return now;
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
		if ( PUSH_SPIN_LIMIT > 1 )
			asm volatile( "{ .reg .pred p; mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
						  : "=r"( done )
						  : "r"( B.barAt ), "r"( parity )
						  : "memory" );
		else /* one look */
			asm volatile( "{ .reg .pred p; mbarrier.test_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
						  : "=r"( done )
						  : "r"( B.barAt ), "r"( parity )
						  : "memory" );
		if ( done || *(volatile int*)&S.gaveUp != 0 )
			return;
		bool late = --left == 0;
		if ( ( left & 255 ) == 0 )
		{
			const unsigned long long now = push_clock();
			start = start == 0 ? now : start;
			late = late || now - start > PUSH_SPIN_NS;
		}
		if ( late )
		{
			for ( int t = 0; t < PUSH_CTAS; ++t )
				*(volatile int*)cg::this_cluster().map_shared_rank( &S.gaveUp, t ) = 1;
			return;
		}
	}
}

/* After the run: no CTA ends before what was sent to it, or by it, is there.  True, on every
 * CTA, when one gave up. */
__device__ __forceinline__ bool push_end( const cg::cluster_group& cl, const PushShared& S )
{
	cl.sync();
	if ( S.gaveUp == 0 )
		return false;
	/* stores that no wait has seen */
	const unsigned long long start = push_clock();
	for ( int left = 1 << 20; push_clock() - start < PUSH_FLIGHT_NS && left > 0; --left )
		;
	cl.sync();
	return true;
}

/* Bytes received in the sweep of a place. */
template <int PHASE, bool JOINTS>
__device__ __forceinline__ int push_bytes( const PushShared& S, int place )
{
	if ( JOINTS && PHASE == F_RESTITUTION )
		return 16 * S.rest[place];
	return 16 * ( PHASE == F_WARM ? S.moved[place] & 0xffff : S.moved[place] >> 16 );
}

template <int PHASE, int T, bool JOINTS>
__device__ __forceinline__ void push_stage( const ResidentPlan& P, const ResShare* share, const SmemRows& m, const ResJoints& J, PushBodies& B,
											PushShared& S, unsigned bars, int sub, const int* ovList, const b2gStepConst& sc )
{
	const int* cs = P.colorStart;
	const int base = 1 + PHASE * B2G_CHAIN_PLACES;
	const int parity = PHASE == F_RESTITUTION ? 0 : sub & 1;
	const int R = cs[B2G_COLORS] - cs[B2G_OVERFLOW];
	const int jointsAll = JOINTS ? P.jointStart[B2G_COLORS] - P.jointStart[B2G_OVERFLOW] : 0;
	const bool colours = PHASE != F_WARM || sc.enableWarmStarting != 0;
	if ( PHASE == F_RESTITUTION ? R > 0 : R + jointsAll > 0 )
	{
		/* without warm starting the overflow set comes next again */
		const int bytes = colours ? push_bytes<PHASE, JOINTS>( S, 0 ) : 0;
		push_expect( B, bars, base, bytes );
		if ( B.rank == 0 )
		{
			const ResShare o = share[B2G_OVERFLOW];
			if ( threadIdx.x == 0 )
			{
				const PushOverflow L{ { B.st0, B.st1 } };
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
			for ( int k = threadIdx.x; k < S.ovCount && colours; k += T )
			{
				const int b = ovList[k], s = b & PUSH_SLOT, t = PUSH_NEXT( b, PHASE );
				if ( t != 0 )
					B.send( B.st0At, s, t, B.st0[s] );
			}
		}
		push_wait( B, S, bytes, parity );
	}
	if ( colours == false )
		return;
	PushStage<PHASE> V;
	(PushBodies&)V = B;
	for ( int a = 0; a < P.activeCount; ++a )
	{
		const int c = P.active[a];
		if ( PHASE == F_RESTITUTION && cs[c + 1] == cs[c] )
			continue;
		const ResShare s = share[c];
		const int bytes = push_bytes<PHASE, JOINTS>( S, 1 + a );
		push_expect( V, bars, base + 1 + a, bytes );
		for ( int j = threadIdx.x; j < s.count; j += T )
			row_step( m, V, s.base + j, PHASE, false, sc );
		if ( JOINTS && PHASE != F_RESTITUTION )
			for ( int i = threadIdx.x; i < s.jcount; i += T )
			{
				b2gJointDev* j = J.at( s.jfirst, s.jbase, i );
				res_joint( j, V, j->indexA, j->indexB, PHASE, sc );
			}
		push_wait( V, S, bytes, parity );
	}
}

/* All substeps; rb: the owned bodies' terms and awake slots, the forwarded ones behind the
 * awake ones.  others: this CTA's copies of other CTAs' bodies. */
template <int T, bool JOINTS>
__device__ __forceinline__ void push_run( const ResidentPlan& P, const ResShare* share, const SmemRows& m, const ResJoints& J, PushBodies& B,
										  PushShared& S, const ResBodies& rb, int awake, int others, const int* ovList, const b2gStepConst& sc )
{
	const unsigned bars = (unsigned)__cvta_generic_to_shared( S.bar );
	const int sent = awake + S.forwards, firstBytes = 16 * S.firsts, restBytes = 16 * S.restFirsts;
	for ( int sub = 0; sub < sc.subSteps; ++sub )
	{
		/* an mbarrier whose wait ran out is not armed again */
		if ( __syncthreads_or( *(volatile int*)&S.gaveUp ) )
			return;
		push_expect( B, bars, 0, firstBytes );
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
			B.pass( s, (int)( B.chain[s].w & 15u ), velocity_word( x ) );
		}
		push_wait( B, S, firstBytes, sub & 1 );
		push_stage<F_WARM, T, JOINTS>( P, share, m, J, B, S, bars, sub, ovList, sc );
		push_stage<F_SOLVE, T, JOINTS>( P, share, m, J, B, S, bars, sub, ovList, sc );
		push_expect( B, bars, PUSH_BAR_POSITION, 16 * others + firstBytes );
		for ( int j = threadIdx.x; j < sent; j += T )
		{
			const int s = rb.awake[j], t = (int)( B.chain[s].w & 15u );
			const float4 v0 = B.st0[s];
			DevState x = state_of( v0, B.st1[s] );
			if ( j < awake )
				integrate_position( x, sc.h );
			const float4 v = make_float4( x.dp.x, x.dp.y, x.dq.c, x.dq.s );
			B.st1[s] = v;
			B.send_position( s, v );
			if ( t != B.rank )
				B.send( B.st0At, s, t, v0 );
		}
		push_wait( B, S, 16 * others + firstBytes, sub & 1 );
		push_stage<F_RELAX, T, JOINTS>( P, share, m, J, B, S, bars, sub, ovList, sc );
	}
	if ( __syncthreads_or( *(volatile int*)&S.gaveUp ) )
		return;
	push_expect( B, bars, PUSH_BAR_RESTITUTION, restBytes );
	for ( int j = threadIdx.x; j < sent; j += T )
	{
		const int s = rb.awake[j], t = (int)( B.chain[s].w >> 4 );
		if ( t != B.rank )
			B.send( B.st0At, s, t, B.st0[s] );
	}
	push_wait( B, S, restBytes, 0 );
	push_stage<F_RESTITUTION, T, JOINTS>( P, share, m, J, B, S, bars, 0, ovList, sc );
}

/* Carves copies after the rows: st0, st1, owned terms and chains, slots, masks, owned ad /
 * flags / awake.  cap copies, of which the first `owned` are the CTA's own bodies. */
__device__ __forceinline__ void push_carve( float4* base, int cap, int owned, int rank, PushBodies& B, ResBodies& rb )
{
	B.st0 = base;
	B.st1 = base + cap;
	rb.st0 = B.st0;
	rb.st1 = B.st1;
	rb.term = base + 2 * cap;
	B.chain = (uint4*)( rb.term + owned );
	B.slot = (unsigned short*)( B.chain + owned );
	B.mask = (unsigned*)( B.slot + PUSH_CTAS * cap );
	rb.ad = (float*)( B.mask + cap );
	rb.flags = (int*)( rb.ad + owned );
	rb.awake = rb.flags + owned;
	B.st0At = (unsigned)__cvta_generic_to_shared( B.st0 );
	B.st1At = (unsigned)__cvta_generic_to_shared( B.st1 );
	B.barAt = 0;
	B.rank = rank;
}

/* Before the CTAs meet for the first time: barriers and counts of this CTA, and of its
 * owned copies the slot, an empty mask and chain.  All threads. */
__device__ __forceinline__ void push_init( PushBodies& B, PushShared& S, const ResidentPlan& P, int owned )
{
	const int tid = threadIdx.x;
	if ( tid == 0 )
	{
		const unsigned bars = (unsigned)__cvta_generic_to_shared( S.bar );
		for ( int i = 0; i < PUSH_BARS; ++i )
			asm volatile( "mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"( bars + 8u * (unsigned)i ) : "memory" );
		asm volatile( "fence.mbarrier_init.release.cluster;" ::: "memory" );
		S.firsts = S.restFirsts = 0;
		S.copies = owned;
		S.fail = S.failAll = S.gaveUp = S.ovCount = S.forwards = 0;
		for ( int a = 0; a < P.activeCount; ++a )
			S.place[P.active[a]] = 1 + a;
		S.place[B2G_OVERFLOW] = 0;
	}
	if ( tid < B2G_CHAIN_PLACES )
		S.moved[tid] = S.rest[tid] = 0;
	for ( int s = tid; s < owned; s += blockDim.x )
	{
		B.mask[s] = 0;
		B.chain[s] = make_uint4( 0, 0, 0, 0 );
		B.slot[PUSH_CTAS * s + B.rank] = (unsigned short)s;
	}
}

/* A body end of a row (or joint) at a place: it joins the body's chain, and the CTA gets a
 * copy the first time it meets the body.  owner, at: where the body lives. */
__device__ __forceinline__ void push_meet( const cg::cluster_group& cl, const PushBodies& B, PushShared& S, int cap, int place, bool row, int owner,
										   int at )
{
	const int rank = B.rank;
	unsigned* chain = (unsigned*)( B.chain + at );
	unsigned* mask = B.mask + at;
	if ( owner != rank )
	{
		chain = cl.map_shared_rank( chain, owner );
		mask = cl.map_shared_rank( mask, owner );
	}
	const unsigned old = atomicOr( chain, 1u << ( place + ( row ? 0 : 16 ) ) );
	if ( place > 0 )
	{
		/* two constraints of one colour on a body have no order */
		if ( ( ( old | old >> 16 ) >> place ) & 1u )
			S.fail = 1;
		if ( rank != 0 )
			atomicOr( chain + 1 + ( place >> 3 ), (unsigned)rank << ( 4 * ( place & 7 ) ) );
	}
	if ( owner == rank )
		return;
	const unsigned bit = 1u << rank;
	if ( atomicOr( mask, bit ) & bit )
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
__device__ __forceinline__ void push_fill( const cg::cluster_group& cl, PushBodies& B, PushShared& S, int owned )
{
	for ( int s = owned + threadIdx.x; s < S.copies; s += blockDim.x )
	{
		const int owner = B.slot[PUSH_CTAS * s], at = B.slot[PUSH_CTAS * s + 1];
		B.st0[s] = *cl.map_shared_rank( B.st0 + at, owner );
		B.st1[s] = *cl.map_shared_rank( B.st1 + at, owner );
		const unsigned m = *cl.map_shared_rank( B.mask + at, owner );
		B.mask[s] = ( m | ( 1u << owner ) ) & ~( 1u << B.rank ) & 0xffffu;
		const uint4* from = cl.map_shared_rank( (const uint4*)( B.slot + PUSH_CTAS * at ), owner );
		uint4* to = (uint4*)( B.slot + PUSH_CTAS * s );
		const uint4 w0 = from[0], w1 = from[1];
		const uint4 w = *cl.map_shared_rank( B.chain + at, owner );
		to[0] = w0;
		to[1] = w1;
		const b2gChain chain = { w.x, { w.y, w.z } };
		if ( b2g_chain_next( chain, -1, 0, 0, owner ) == B.rank )
			atomicAdd( &S.firsts, 1 );
		if ( b2g_chain_next( chain, -1, 0, 1, owner ) == B.rank )
			atomicAdd( &S.restFirsts, 1 );
	}
}

/* This CTA's copy of a body with the CTAs that need it after the place. */
__device__ __forceinline__ int push_take( const cg::cluster_group& cl, const PushBodies& B, int place, int owner, int at )
{
	const int rank = B.rank;
	const int s = owner == rank ? at : (int)*cl.map_shared_rank( B.slot + PUSH_CTAS * at + rank, owner );
	const uint4 w = owner == rank ? B.chain[at] : *cl.map_shared_rank( B.chain + at, owner );
	const b2gChain chain = { w.x, { w.y, w.z } };
	const int warm = b2g_chain_next( chain, place, 1, 0, owner );
	const int solve = b2g_chain_next( chain, place, 0, 0, owner );
	/* a body that no row moves here is nobody's in restitution */
	const int rest = ( ( chain.who >> place ) & 1u ) ? b2g_chain_next( chain, place, 0, 1, owner ) : rank;
	return s | warm << 16 | solve << 20 | rest << 24;
}

/* Tells the CTAs that receive body b (slot and next CTAs) after a place; overflow bodies are
 * told once, and listed. */
template <bool JOINTS>
__device__ __forceinline__ void push_count( const cg::cluster_group& cl, const PushBodies& B, PushShared& S, int b, int place, int* ovList )
{
	if ( place == 0 )
	{
		if ( atomicOr( B.mask + ( b & PUSH_SLOT ), PUSH_LISTED ) & PUSH_LISTED )
			return;
		ovList[atomicAdd( &S.ovCount, 1 )] = b;
	}
	const int warm = PUSH_NEXT( b, F_WARM ), solve = PUSH_NEXT( b, F_SOLVE ), rest = PUSH_NEXT( b, F_RESTITUTION );
	if ( warm != B.rank )
		atomicAdd( cl.map_shared_rank( S.moved + place, warm ), solve == warm ? 0x10001 : 1 );
	if ( solve != B.rank && solve != warm )
		atomicAdd( cl.map_shared_rank( S.moved + place, solve ), 0x10000 );
	if ( JOINTS && rest != B.rank )
		atomicAdd( cl.map_shared_rank( S.rest + place, rest ), 1 );
}

/* From rows and joints on body ids to rows and joints on copies, with the expected bytes
 * counted; false, on every CTA, when a CTA's copies do not fit (or two constraints of one
 * colour share a body): the ids are unchanged then.  Owned bodies (of block ids a CTA, inv
 * its reciprocal) are in the first slots of their owners; behind the `awake` ones of
 * rb.awake, which integrated( s ) knows, come the others with copies elsewhere.  All threads
 * of the cluster; the caller meets the other CTAs before the first sweep. */
template <bool JOINTS, class F>
__device__ __forceinline__ bool push_exchange( const cg::cluster_group& cl, PushBodies& B, PushShared& S, int cap, int block, unsigned inv, int rows,
											   int joints, const ResShare* share, const SmemRows& m, const ResJoints& J, int* ovList,
											   const ResBodies& rb, const int& awake, F integrated )
{
	const int tid = threadIdx.x, T = blockDim.x;
	auto owner_of = [&]( int b ) { return block == 1 ? b : (int)__umulhi( (unsigned)b, inv ); };
	auto meet = [&]( int b, int c, bool row ) {
		if ( b >= 0 )
			push_meet( cl, B, S, cap, S.place[c], row, owner_of( b ), b - owner_of( b ) * block );
	};
	auto take = [&]( int b, int c ) {
		if ( b < 0 )
			return -1;
		b = push_take( cl, B, S.place[c], owner_of( b ), b - owner_of( b ) * block );
		push_count<JOINTS>( cl, B, S, b, S.place[c], ovList );
		return b;
	};
	auto row_at = [&]( int k, int& c ) {
		while ( k >= share[c].base + share[c].count )
			++c;
	};
	auto joint_at = [&]( int k, int& c ) {
		while ( k >= share[c].jbase + share[c].jcount )
			++c;
		return J.at( share[c].jfirst, share[c].jbase, k - share[c].jbase );
	};
	cl.sync();
	for ( int k = tid, c = 0; k < rows; k += T )
	{
		row_at( k, c );
		meet( m.idx[k].x, c, true );
		meet( m.idx[k].y, c, true );
	}
	if ( JOINTS )
		for ( int k = tid, c = 0; k < joints; k += T )
		{
			const b2gJointDev* j = joint_at( k, c );
			meet( j->indexA, c, false );
			meet( j->indexB, c, false );
		}
	__syncthreads();
	if ( tid < PUSH_CTAS && S.fail )
		*cl.map_shared_rank( &S.failAll, tid ) = 1;
	cl.sync();
	if ( S.failAll )
		return false;
	push_fill( cl, B, S, block );
	for ( int s = tid; s < block; s += T )
		if ( ( B.mask[s] & 0xffffu ) != 0 && integrated( s ) == false )
			rb.awake[awake + atomicAdd( &S.forwards, 1 )] = s;
	__syncthreads();
	for ( int k = tid, c = 0; k < rows; k += T )
	{
		row_at( k, c );
		const int4 ix = m.idx[k];
		m.idx[k].x = take( ix.x, c );
		m.idx[k].y = take( ix.y, c );
	}
	if ( JOINTS )
		for ( int k = tid, c = 0; k < joints; k += T )
		{
			b2gJointDev* j = joint_at( k, c );
			j->indexA = take( j->indexA, c );
			j->indexB = take( j->indexB, c );
		}
	/* read by the owner alone */
	for ( int j = tid; j < awake + S.forwards; j += T )
	{
		const int s = rb.awake[j];
		const b2gChain chain = { B.chain[s].x, { B.chain[s].y, B.chain[s].z } };
		B.chain[s].w = (unsigned)( b2g_chain_next( chain, -1, 0, 0, B.rank ) | b2g_chain_next( chain, -1, 0, 1, B.rank ) << 4 );
	}
	return true;
}
