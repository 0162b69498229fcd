/*
 * give_up_check.cu -- a contact solve whose waits run out marks its result: built with
 * limits of one poll (-DPUSH_SPIN_LIMIT=1 -DRES_SPIN_LIMIT=1), a cluster and a grid give up
 * at the first wait that another CTA has not met yet.  Every listed body then has NaN
 * velocities, the context stays usable, and a second call gives the same.  Prints
 * "status no error" at the end.
 */
#include "box2d/gpu.h"

#include <cuda_runtime.h>

#include <cmath>
#include <stdio.h>
#include <string.h>
#include <vector>

/* Rows of n bodies in a chain, contacts of even and odd links in two colours, and `overflow`
 * of the last links in the overflow set. */
static int run( const char* name, int n, int overflow )
{
	std::vector<float> states( 8 * (size_t)n, 0.0f ), mass( 4 * (size_t)n, 1.0f ), forces( 4 * (size_t)n, 0.0f ), damping( 4 * (size_t)n, 0.0f );
	std::vector<int> bodies( (size_t)n ), pairs;
	for ( int i = 0; i < n; ++i )
	{
		states[8 * i] = 0.01f * ( i % 7 );
		states[8 * i + 6] = 1.0f;
		bodies[i] = i;
	}
	b2ContactSolveDesc d;
	memset( &d, 0, sizeof( d ) );
	const int links = n - 1, coloured = links - overflow;
	for ( int c = 0; c < 2; ++c )
	{
		d.colorStart[c] = (int)pairs.size() / 2;
		for ( int i = c; i < coloured; i += 2 )
		{
			pairs.push_back( i );
			pairs.push_back( i + 1 );
		}
	}
	for ( int c = 2; c < 12; ++c )
		d.colorStart[c] = (int)pairs.size() / 2;
	for ( int i = coloured; i < links; ++i )
	{
		pairs.push_back( i );
		pairs.push_back( i + 1 );
	}
	d.colorStart[12] = (int)pairs.size() / 2;
	const int contacts = d.colorStart[12];
	std::vector<float> mix( 2 * (size_t)contacts, 0.5f );
	std::vector<b2Manifold> manifolds( (size_t)contacts );
	memset( manifolds.data(), 0, sizeof( b2Manifold ) * manifolds.size() );
	for ( b2Manifold& m : manifolds )
	{
		m.normal = { 1.0f, 0.0f };
		m.pointCount = 1;
		m.points[0].anchorA = { 0.5f, 0.0f };
		m.points[0].anchorB = { -0.5f, 0.0f };
	}
	struct Copy
	{
		const void* from;
		size_t bytes;
		void* to;
	} copies[] = { { states.data(), 4 * states.size(), nullptr },	 { mass.data(), 4 * mass.size(), nullptr },
				   { forces.data(), 4 * forces.size(), nullptr },	 { damping.data(), 4 * damping.size(), nullptr },
				   { bodies.data(), 4 * bodies.size(), nullptr },	 { pairs.data(), 4 * pairs.size(), nullptr },
				   { mix.data(), 4 * mix.size(), nullptr },			 { manifolds.data(), sizeof( b2Manifold ) * manifolds.size(), nullptr } };
	for ( Copy& c : copies )
	{
		cudaMalloc( &c.to, c.bytes );
		cudaMemcpy( c.to, c.from, c.bytes, cudaMemcpyHostToDevice );
	}
	d.states = (float*)copies[0].to;
	d.massData = (const float*)copies[1].to;
	d.forces = (const float*)copies[2].to;
	d.damping = (const float*)copies[3].to;
	d.bodies = (const int*)copies[4].to;
	d.bodyCount = n;
	d.contactBodies = (const int*)copies[5].to;
	d.contactMix = (const float*)copies[6].to;
	d.manifolds = (b2Manifold*)copies[7].to;
	d.contactCount = contacts;
	d.timeStep = 1.0f / 60.0f;
	d.subStepCount = 4;
	d.gravity = { 0.0f, -10.0f };
	d.contactHertz = 30.0f;
	d.contactDampingRatio = 10.0f;
	d.contactPushout = 3.0f;
	d.restitutionThreshold = 1.0f;
	d.enableWarmStarting = true;
	int bad = 0;
	for ( int call = 0; call < 2; ++call )
	{
		cudaMemcpy( copies[0].to, copies[0].from, copies[0].bytes, cudaMemcpyHostToDevice );
		int rc = b2SolveContacts( &d );
		cudaError_t e = cudaDeviceSynchronize();
		std::vector<float> out( states.size() );
		cudaMemcpy( out.data(), copies[0].to, copies[0].bytes, cudaMemcpyDeviceToHost );
		int marked = 0;
		for ( int i = 0; i < n; ++i )
			marked += std::isnan( out[8 * i] ) && std::isnan( out[8 * i + 1] ) && std::isnan( out[8 * i + 2] );
		printf( "%s: %d contacts, call %d: rc %d, %s, %d of %d bodies marked\n", name, contacts, call, rc, cudaGetErrorString( e ), marked, n );
		if ( rc != 0 || e != cudaSuccess || marked != n )
		{
			printf( "MISMATCH\n" );
			bad = 1;
		}
	}
	for ( Copy& c : copies )
		cudaFree( c.to );
	return bad;
}

int main()
{
	int bad = run( "cluster", 4000, 200 );
	bad |= run( "grid", 60000, 0 );
	bad |= run( "grid with rows in memory", 12000, 3000 );
	printf( "status %s\n", cudaGetErrorString( cudaGetLastError() ) );
	return bad;
}
