/*
 * b2g_chain.h -- the order in which the constraints of a cluster move one body, and so the
 * CTA that needs the body's velocity next (b2g_push.h).
 *
 * Place 0 of a stage is the overflow set, place 1 + a the stage's a-th active colour.  At
 * most one row or joint of a colour moves a body (src/constraint_graph.c:84-131), and all
 * overflow constraints are CTA 0's, so a place is moved by one CTA or by none.
 */
#pragma once

#ifdef __CUDACC__
#define B2G_CHAIN_FN static __host__ __device__ __forceinline__
#else
#define B2G_CHAIN_FN static inline
#endif

#define B2G_CHAIN_PLACES 12
#define B2G_CHAIN_NONE 16

/* who: bit p a row at place p, bit 16 + p a joint; cta: four bits a place. */
typedef struct b2gChain
{
	unsigned who, cta[2];
} b2gChain;

/* The places of a stage: all constraints, or in restitution the rows. */
B2G_CHAIN_FN unsigned b2g_chain_places( b2gChain c, int restitution ) { return ( restitution ? c.who : c.who | c.who >> 16 ) & 0xfffu; }

/* The CTA at the first of the places after p (-1: at the first), or B2G_CHAIN_NONE. */
B2G_CHAIN_FN int b2g_chain_after( b2gChain c, unsigned places, int p )
{
	for ( int q = p + 1; q < B2G_CHAIN_PLACES; ++q )
		if ( ( places >> q ) & 1u )
			return (int)( ( q < 8 ? c.cta[0] >> ( 4 * q ) : c.cta[1] >> ( 4 * q - 32 ) ) & 15u );
	return B2G_CHAIN_NONE;
}

/* The CTA that needs the velocity after place p (-1: after an integration, or at the start
 * of restitution).  After a warm start comes the first place again; after every other stage
 * the owner, which integrates the velocity, the position or the body's end of step. */
B2G_CHAIN_FN int b2g_chain_next( b2gChain c, int p, int warm, int restitution, int owner )
{
	unsigned places = b2g_chain_places( c, restitution );
	int t = b2g_chain_after( c, places, p );
	if ( t == B2G_CHAIN_NONE && warm )
		t = b2g_chain_after( c, places, -1 );
	return t == B2G_CHAIN_NONE ? owner : t;
}
