/*
 * The register narrowphase (b2g_collide_small.h) against the general one (b2g_collide.h)
 * on random shape pairs near contact: circles, capsules, segments, polygons of three to
 * eight vertices, rounded or not, and degenerate placements.  Built and run by
 * tests/test_gpu_narrowphase.py; prints the pairs compared and MISMATCH lines.
 */
#include "b2g_stages.h"

#include <stdio.h>
#include <stdlib.h>
#include <vector>

struct Pair
{
	b2gShapeGeo a, b;
	b2gXf xfA, xfB;
};

__global__ void k_both( const Pair* pairs, int n, b2gManifold* small, b2gManifold* general, int* handled )
{
	int i = blockIdx.x * blockDim.x + threadIdx.x;
	if ( i >= n )
		return;
	const Pair& p = pairs[i];
	b2gManifold m;
	handled[i] = small_narrowphase( m, &p.a, p.xfA, &p.b, p.xfB ) ? 1 : 0;
	small[i] = m;
	uint32_t cache = 0;
	general[i] = narrowphase_general( &p.a, p.xfA, &p.b, p.xfB, &cache );
}

static float frand( float lo, float hi ) { return lo + ( hi - lo ) * (float)( rand() / ( RAND_MAX + 1.0 ) ); }

static b2gShapeGeo shape( int type, int count )
{
	b2gShapeGeo g;
	memset( &g, 0, sizeof( g ) );
	g.type = type;
	g.radius = type == 2 ? 0.0f : ( type == 3 ? ( rand() & 1 ? 0.0f : frand( 0.01f, 0.2f ) ) : frand( 0.1f, 0.5f ) );
	if ( type != 3 )
	{
		g.v[0] = gv( frand( -0.5f, 0.5f ), frand( -0.5f, 0.5f ) );
		g.v[1] = gv( frand( -0.5f, 0.5f ), frand( -0.5f, 0.5f ) );
		return g;
	}
	g.count = count;
	float ex = frand( 0.3f, 0.8f ), ey = frand( 0.3f, 0.8f ), at = frand( 0.0f, 1.0f );
	bool box = count == 4 && ( rand() & 1 );
	for ( int i = 0; i < count; ++i )
	{
		float t = 6.2831853f * ( (float)i + ( box ? 0.5f : at ) ) / (float)count;
		g.v[i] = box ? gv( i == 0 || i == 3 ? 0.5f : -0.5f, i < 2 ? 0.5f : -0.5f ) : gv( ex * cosf( t ), ey * sinf( t ) );
	}
	for ( int i = 0; i < count; ++i )
		g.n[i] = gnormalize( gright( gsub( g.v[( i + 1 ) % count], g.v[i] ) ) );
	return g;
}

int main( void )
{
	srand( 7 );
	const int n = 300000;
	std::vector<Pair> pairs( n );
	for ( int i = 0; i < n; ++i )
	{
		/* the narrowphase's orders: the higher type first, capsules also against segments */
		int types[2] = { rand() % 4, rand() % 4 };
		if ( types[0] < types[1] )
			std::swap( types[0], types[1] );
		if ( types[0] == 2 && types[1] == 2 )
			types[1] = 1;
		Pair& p = pairs[i];
		p.a = shape( types[0], 3 + rand() % ( i % 4 == 0 ? 6 : 2 ) );
		p.b = shape( types[1], 3 + rand() % ( i % 4 == 0 ? 6 : 2 ) );
		float a = i % 5 == 0 ? 0.0f : frand( -3.2f, 3.2f ), b = i % 5 == 0 ? 0.0f : frand( -3.2f, 3.2f );
		p.xfA.p = gv( frand( -5.0f, 5.0f ), frand( -5.0f, 5.0f ) );
		p.xfA.q = grot( cosf( a ), sinf( a ) );
		float d = i % 7 == 0 ? 1.0f : frand( 0.0f, 1.6f ), t = i % 5 == 0 ? 1.5707963f * (float)( rand() % 4 ) : frand( -3.2f, 3.2f );
		p.xfB.p = gv( p.xfA.p.x + d * cosf( t ), p.xfA.p.y + d * sinf( t ) );
		p.xfB.q = grot( cosf( b ), sinf( b ) );
	}
	Pair* dp;
	b2gManifold *ds, *dg;
	int* dh;
	cudaMalloc( &dp, sizeof( Pair ) * n );
	cudaMalloc( &ds, sizeof( b2gManifold ) * n );
	cudaMalloc( &dg, sizeof( b2gManifold ) * n );
	cudaMalloc( &dh, sizeof( int ) * n );
	cudaMemcpy( dp, pairs.data(), sizeof( Pair ) * n, cudaMemcpyHostToDevice );
	k_both<<<( n + 127 ) / 128, 128>>>( dp, n, ds, dg, dh );
	std::vector<b2gManifold> s( n ), g( n );
	std::vector<int> h( n );
	cudaMemcpy( s.data(), ds, sizeof( b2gManifold ) * n, cudaMemcpyDeviceToHost );
	cudaMemcpy( g.data(), dg, sizeof( b2gManifold ) * n, cudaMemcpyDeviceToHost );
	cudaMemcpy( h.data(), dh, sizeof( int ) * n, cudaMemcpyDeviceToHost );
	printf( "status %s\n", cudaGetErrorString( cudaGetLastError() ) );
	int compared = 0, touching[3] = { 0, 0, 0 }, bad = 0;
	for ( int i = 0; i < n; ++i )
	{
		const Pair& p = pairs[i];
		bool fits = ( p.a.type != 3 || p.a.count <= 4 ) && ( p.b.type != 3 || p.b.count <= 4 );
		/* a circle needs the other shape's count only when that is a polygon */
		if ( h[i] != ( fits ? 1 : 0 ) && bad++ < 10 )
			printf( "MISMATCH pair %d: handled %d\n", i, h[i] );
		if ( h[i] == 0 )
			continue;
		compared += 1;
		touching[g[i].count] += 1;
		/* fields, not padding */
		bool same = s[i].count == g[i].count && memcmp( &s[i].normal, &g[i].normal, sizeof( b2gVec ) ) == 0;
		for ( int j = 0; j < 2; ++j )
			same = same && memcmp( s[i].pts + j, g[i].pts + j, offsetof( b2gPoint, pad ) ) == 0;
		if ( same == false && bad++ < 10 )
			printf( "MISMATCH pair %d: types %d %d counts %d %d\n", i, p.a.type, p.b.type, s[i].count, g[i].count );
	}
	printf( "compared %d touching %d %d %d\n", compared, touching[0], touching[1], touching[2] );
	return bad != 0;
}
