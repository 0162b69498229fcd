/*
 * b2g_collide_small.h -- manifolds of polygons of at most four vertices, and of capsules
 * and segments as rounded 2-gons, in registers.
 *
 * The functions of b2g_collide.h index their vertex arrays at run time, which puts them in
 * local memory: a box pair walks about 900 bytes of it in dependent loads and stores.
 * Nearly every shape of a scene has four vertices or fewer; for those every loop here has
 * constant bounds, an edge found at run time is picked by comparison, and nothing leaves
 * the registers.  Each expression is that of b2g_collide.h (reference src/manifold.c:14-30,
 * :183-270, :276-700), so the manifolds are the same bits.
 *
 * Narrowphase of a step, launch included, general path before and this one now: 590 box
 * pairs 17 -> 12 us, 15000 19 -> 13.5, 58000 28 -> 19; 2000 pairs of boxes, circles and
 * capsules 34 -> 21; 1024 batched pyramids (950000 pairs) 300 -> 240 us.
 */
#pragma once

#include "b2g_collide.h"

#define SMALL_MAX 4

struct SmallPoly
{
	b2gVec v[SMALL_MAX], n[SMALL_MAX];
	int count;
	float radius;
};

__device__ __forceinline__ b2gVec small_pick( const b2gVec* a, int i )
{
	b2gVec r = a[0];
#pragma unroll
	for ( int k = 1; k < SMALL_MAX; ++k )
	{
		r.x = i == k ? a[k].x : r.x;
		r.y = i == k ? a[k].y : r.y;
	}
	return r;
}

/* Vertices and normals of a shape that is no circle or chain link; false when it has more
 * than SMALL_MAX.  Shape records are 160 bytes apart on a 16-byte boundary, vertices at
 * byte 16 and normals at 80. */
__device__ __forceinline__ bool small_shape( SmallPoly& p, const b2gShapeGeo* g )
{
	const float4* v4 = (const float4*)g->v;
	if ( g->type == 3 )
	{
		if ( g->count > SMALL_MAX )
			return false;
		const float4* n4 = (const float4*)g->n;
		float4 a = v4[0], b = v4[1], c = n4[0], d = n4[1];
		p.v[0] = gv( a.x, a.y );
		p.v[1] = gv( a.z, a.w );
		p.v[2] = gv( b.x, b.y );
		p.v[3] = gv( b.z, b.w );
		p.n[0] = gv( c.x, c.y );
		p.n[1] = gv( c.z, c.w );
		p.n[2] = gv( d.x, d.y );
		p.n[3] = gv( d.z, d.w );
		p.count = g->count;
		p.radius = g->radius;
		return true;
	}
	/* gmake_capsule */
	float4 a = v4[0];
	p.v[0] = gv( a.x, a.y );
	p.v[1] = gv( a.z, a.w );
	b2gVec axis = gnormalize( gsub( p.v[1], p.v[0] ) );
	b2gVec normal = gright( axis );
	p.n[0] = normal;
	p.n[1] = gneg( normal );
	p.v[2] = p.v[3] = p.n[2] = p.n[3] = gv( 0.0f, 0.0f );
	p.count = 2;
	p.radius = g->type == 1 ? g->radius : 0.0f;
	return true;
}

__device__ __forceinline__ float small_max_separation( int& edge, const SmallPoly& p1, const SmallPoly& p2 )
{
	int best = 0;
	float maxSep = -FLT_MAX;
#pragma unroll
	for ( int i = 0; i < SMALL_MAX; ++i )
	{
		b2gVec n = p1.n[i];
		b2gVec v1 = p1.v[i];
		float si = FLT_MAX;
#pragma unroll
		for ( int j = 0; j < SMALL_MAX; ++j )
		{
			float sij = gdot( n, gsub( p2.v[j], v1 ) );
			if ( j < p2.count && sij < si )
				si = sij;
		}
		if ( i < p1.count && si > maxSep )
		{
			maxSep = si;
			best = i;
		}
	}
	edge = best;
	return maxSep;
}

/* The edge of p most against `search`. */
__device__ __forceinline__ int small_opposite( b2gVec search, const SmallPoly& p )
{
	int edge = 0;
	float minDot = FLT_MAX;
#pragma unroll
	for ( int i = 0; i < SMALL_MAX; ++i )
	{
		float d = gdot( search, p.n[i] );
		if ( i < p.count && d < minDot )
		{
			minDot = d;
			edge = i;
		}
	}
	return edge;
}

/* gclip_polygons on the chosen edges: v11 v12 with its normal the reference edge of
 * polygon 1, v21 v22 the incident edge of polygon 2. */
__device__ __forceinline__ void small_clip( b2gManifold& m, b2gVec normal, b2gVec v11, b2gVec v12, b2gVec v21, b2gVec v22, float r1, float r2,
											int i11, int i12, int i21, int i22, bool flip )
{
	b2gVec tangent = gcross_sv( 1.0f, normal );
	float lower1 = 0.0f;
	float upper1 = gdot( gsub( v12, v11 ), tangent );
	float upper2 = gdot( gsub( v21, v11 ), tangent );
	float lower2 = gdot( gsub( v22, v11 ), tangent );
	b2gVec vLower, vUpper;
	if ( lower2 < lower1 && upper2 - lower2 > FLT_EPSILON )
		vLower = glerp( v22, v21, ( lower1 - lower2 ) / ( upper2 - lower2 ) );
	else
		vLower = v22;
	if ( upper2 > upper1 && upper2 - lower2 > FLT_EPSILON )
		vUpper = glerp( v22, v21, ( upper1 - lower2 ) / ( upper2 - lower2 ) );
	else
		vUpper = v21;
	float sepLower = gdot( gsub( vLower, v11 ), normal );
	float sepUpper = gdot( gsub( vUpper, v11 ), normal );
	vLower = gmuladd( vLower, 0.5f * ( r1 - r2 - sepLower ), normal );
	vUpper = gmuladd( vUpper, 0.5f * ( r1 - r2 - sepUpper ), normal );
	float radius = r1 + r2;
	m.normal = flip ? gneg( normal ) : normal;
	m.pts[0].anchorA = flip ? vUpper : vLower;
	m.pts[0].separation = ( flip ? sepUpper : sepLower ) - radius;
	m.pts[0].id = flip ? B2G_MAKE_ID( i21, i12 ) : B2G_MAKE_ID( i11, i22 );
	m.pts[1].anchorA = flip ? vLower : vUpper;
	m.pts[1].separation = ( flip ? sepLower : sepUpper ) - radius;
	m.pts[1].id = flip ? B2G_MAKE_ID( i22, i11 ) : B2G_MAKE_ID( i12, i21 );
	m.count = 2;
}

/* gcollide_polygons_raw */
__device__ __forceinline__ void small_polygons( b2gManifold& m, const SmallPoly& inA, b2gXf xfA, const SmallPoly& inB, b2gXf xfB )
{
	b2gVec origin = inA.v[0];
	b2gXf sfA;
	sfA.p = gadd( xfA.p, grotate( xfA.q, origin ) );
	sfA.q = xfA.q;
	b2gXf xf = ginvmulxf( sfA, xfB );
	SmallPoly A, B;
	A.count = inA.count;
	A.radius = inA.radius;
	A.v[0] = gv( 0.0f, 0.0f );
	A.n[0] = inA.n[0];
#pragma unroll
	for ( int i = 1; i < SMALL_MAX; ++i )
	{
		A.v[i] = gsub( inA.v[i], origin );
		A.n[i] = inA.n[i];
	}
	B.count = inB.count;
	B.radius = inB.radius;
#pragma unroll
	for ( int i = 0; i < SMALL_MAX; ++i )
	{
		B.v[i] = gxfpoint( xf, inB.v[i] );
		B.n[i] = grotate( xf.q, inB.n[i] );
	}

	int edgeA, edgeB;
	float sepA = small_max_separation( edgeA, A, B );
	float sepB = small_max_separation( edgeB, B, A );
	float radius = A.radius + B.radius;
	if ( sepA > B2G_SPECULATIVE + radius || sepB > B2G_SPECULATIVE + radius )
		return;
	const bool flip = !( sepA >= sepB );
	if ( flip == false )
		edgeB = small_opposite( small_pick( A.n, edgeA ), B );
	else
		edgeA = small_opposite( small_pick( B.n, edgeB ), A );

	const int a1 = edgeA, a2 = edgeA + 1 < A.count ? edgeA + 1 : 0;
	const int b1 = edgeB, b2 = edgeB + 1 < B.count ? edgeB + 1 : 0;
	const b2gVec va1 = small_pick( A.v, a1 ), va2 = small_pick( A.v, a2 );
	const b2gVec vb1 = small_pick( B.v, b1 ), vb2 = small_pick( B.v, b2 );
	bool clip = true;
	if ( sepA > 0.1f * B2G_LINEAR_SLOP || sepB > 0.1f * B2G_LINEAR_SLOP )
	{
		b2gSegDist r = gsegment_distance( va1, va2, vb1, vb2 );
		const bool end1 = r.f1 == 0.0f || r.f1 == 1.0f, end2 = r.f2 == 0.0f || r.f2 == 1.0f;
		if ( end1 && end2 )
		{
			/* two vertices are nearest */
			clip = false;
			const bool first1 = r.f1 == 0.0f, first2 = r.f2 == 0.0f;
			b2gVec vA = first1 ? va1 : va2, vB = first2 ? vb1 : vb2;
			b2gVec normal = gsub( vB, vA );
			float distance = sqrtf( r.dist2 );
			if ( distance > B2G_SPECULATIVE + radius )
				return;
			float inv = 1.0f / distance;
			normal.x *= inv;
			normal.y *= inv;
			b2gVec c1 = gmuladd( vA, A.radius, normal );
			b2gVec c2 = gmuladd( vB, -B.radius, normal );
			m.normal = normal;
			m.pts[0].anchorA = glerp( c1, c2, 0.5f );
			m.pts[0].separation = distance - radius;
			m.pts[0].id = B2G_MAKE_ID( first1 ? a1 : a2, first2 ? b1 : b2 );
			m.count = 1;
		}
	}
	if ( clip )
	{
		b2gVec nA = small_pick( A.n, a1 ), nB = small_pick( B.n, b1 );
		if ( flip )
			small_clip( m, nB, vb1, vb2, va1, va2, B.radius, A.radius, b1, b2, a1, a2, true );
		else
			small_clip( m, nA, va1, va2, vb1, vb2, A.radius, B.radius, a1, a2, b1, b2, false );
	}

	m.normal = grotate( xfA.q, m.normal );
#pragma unroll
	for ( int i = 0; i < 2; ++i )
	{
		if ( i < m.count )
		{
			m.pts[i].anchorA = grotate( xfA.q, gadd( m.pts[i].anchorA, origin ) );
			m.pts[i].anchorB = gadd( m.pts[i].anchorA, gsub( xfA.p, xfB.p ) );
			m.pts[i].point = gadd( xfA.p, m.pts[i].anchorA );
		}
	}
}

/* gcollide_polygon_circle */
__device__ __forceinline__ void small_polygon_circle( b2gManifold& m, const SmallPoly& a, b2gXf xfA, b2gVec centerB, float rB, b2gXf xfB )
{
	b2gXf xf = ginvmulxf( xfA, xfB );
	b2gVec c = gxfpoint( xf, centerB );
	float rA = a.radius;
	float radius = rA + rB;
	int i1 = 0;
	float separation = -FLT_MAX;
#pragma unroll
	for ( int i = 0; i < SMALL_MAX; ++i )
	{
		float s = gdot( a.n[i], gsub( c, a.v[i] ) );
		if ( i < a.count && s > separation )
		{
			separation = s;
			i1 = i;
		}
	}
	if ( separation > radius + B2G_SPECULATIVE )
		return;
	int i2 = i1 + 1 < a.count ? i1 + 1 : 0;
	b2gVec v1 = small_pick( a.v, i1 ), v2 = small_pick( a.v, i2 );
	float u1 = gdot( gsub( c, v1 ), gsub( v2, v1 ) );
	float u2 = gdot( gsub( c, v2 ), gsub( v1, v2 ) );
	const bool at1 = u1 < 0.0f && separation > FLT_EPSILON;
	const bool at2 = u2 < 0.0f && separation > FLT_EPSILON;
	if ( at1 || at2 )
	{
		b2gVec v = at1 ? v1 : v2;
		b2gVec normal = gnormalize( gsub( c, v ) );
		separation = gdot( gsub( c, v ), normal );
		if ( separation > radius + B2G_SPECULATIVE )
			return;
		b2gVec cA = gmuladd( v, rA, normal );
		b2gVec cB = gmulsub( c, rB, normal );
		gone_point( &m, xfA, xfB, normal, glerp( cA, cB, 0.5f ), gdot( gsub( cB, cA ), normal ) );
	}
	else
	{
		b2gVec normal = small_pick( a.n, i1 );
		b2gVec cA = gmuladd( c, rA - gdot( gsub( c, v1 ), normal ), normal );
		b2gVec cB = gmulsub( c, rB, normal );
		gone_point( &m, xfA, xfB, normal, glerp( cA, cB, 0.5f ), separation - radius );
	}
}

/* The narrowphase of two shapes that are no sensors; false when one of them needs the
 * general path (a chain link, a polygon of more than SMALL_MAX vertices). */
__device__ __forceinline__ bool small_narrowphase( b2gManifold& m, const b2gShapeGeo* gA, b2gXf xfA, const b2gShapeGeo* gB, b2gXf xfB )
{
	gmanifold_clear( &m );
	const int tA = gA->type, tB = gB->type;
	if ( tA == 4 )
		return false;
	if ( tB == 0 && tA != 3 )
	{
		if ( tA == 0 )
			gcollide_circles( &m, gA->v[0], gA->radius, xfA, gB->v[0], gB->radius, xfB );
		else
			gcollide_capsule_circle( &m, gA->v[0], gA->v[1], tA == 1 ? gA->radius : 0.0f, xfA, gB->v[0], gB->radius, xfB );
		return true;
	}
	SmallPoly A;
	if ( small_shape( A, gA ) == false )
		return false;
	if ( tB == 0 )
	{
		small_polygon_circle( m, A, xfA, gB->v[0], gB->radius, xfB );
		return true;
	}
	SmallPoly B;
	if ( small_shape( B, gB ) == false )
		return false;
	small_polygons( m, A, xfA, B, xfB );
	return true;
}
