/*
 * adjoint_memory.c -- the backward call's device memory (box2c_gb300/csrc/adjoint.c) against
 * a runtime that has only so much: it replays as many steps at a time as there is memory
 * for, down to one, fails below that and works afterwards, and gives its memory back
 * with the last tape.  Prints "ok" or the first failure.
 */
#include "host.h"

#include "box2d/gpu.h"

#include <cuda_runtime_api.h>

#include <stdio.h>
#include <stdlib.h>
#include <string.h>

/* ------------------------------------------------------------------ a runtime of s_limit bytes */
static size_t s_limit, s_used;
static int s_error, s_streams;

cudaError_t cudaMalloc( void** p, size_t n )
{
	if ( s_used + n > s_limit )
	{
		s_error = cudaErrorMemoryAllocation;
		return cudaErrorMemoryAllocation;
	}
	size_t* b = malloc( n + 16 );
	*b = n;
	s_used += n;
	*p = (char*)b + 16;
	return cudaSuccess;
}
cudaError_t cudaFree( void* p )
{
	if ( p )
	{
		s_used -= *(size_t*)( (char*)p - 16 );
		free( (char*)p - 16 );
	}
	return cudaSuccess;
}
cudaError_t cudaMallocHost( void** p, size_t n )
{
	*p = malloc( n );
	return cudaSuccess;
}
cudaError_t cudaFreeHost( void* p )
{
	free( p );
	return cudaSuccess;
}
cudaError_t cudaGetLastError( void )
{
	int e = s_error;
	s_error = 0;
	return e;
}
cudaError_t cudaMemcpyAsync( void* d, const void* s, size_t n, enum cudaMemcpyKind k, cudaStream_t t )
{
	memcpy( d, s, n );
	return cudaSuccess;
}
cudaError_t cudaMemcpy( void* d, const void* s, size_t n, enum cudaMemcpyKind k )
{
	memcpy( d, s, n );
	return cudaSuccess;
}
cudaError_t cudaMemsetAsync( void* d, int v, size_t n, cudaStream_t t )
{
	memset( d, v, n );
	return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags( cudaStream_t* s, unsigned f )
{
	s_streams += 1;
	*s = (cudaStream_t)&s_streams;
	return cudaSuccess;
}
cudaError_t cudaStreamSynchronize( cudaStream_t s ) { return cudaSuccess; }
cudaError_t cudaDeviceSynchronize( void ) { return cudaSuccess; }

/* ------------------------------------------------------------------ worlds and kernels */
#define STEP_FLOATS 100000u
#define CARRIED_FLOATS 1000u

static gWorld s_worlds[2];
static gShape s_shape;
static int s_chunk, s_launches;

void* b2g_calloc( size_t n, size_t size ) { return calloc( n, size ); }
void* b2g_realloc( void* p, size_t n ) { return realloc( p, n ); }
void b2g_free( void* p ) { free( p ); }
bool b2World_IsValid( b2WorldId id ) { return true; }
gWorld* gworld_get( b2WorldId id ) { return s_worlds + id.index1; }
int b2gd_tape_record( b2gDevWorld* w, void* bodies, int bodyCount, void* rows, int rowCount ) { return 0; }
size_t b2gd_adjoint_scratch( int bodies, int rows, int chunk ) { return CARRIED_FLOATS + (size_t)chunk; }
size_t b2gd_adjoint_step_scratch( int bodies, int rows, int contacts, int sub ) { return STEP_FLOATS; }
int b2gd_adjoint_launch( const b2gAdjointItem* items, int count, int steps, int chunk, int bodies, int rows, int sub, void* stream )
{
	/* every world's scratch is its own, and inside an allocation */
	for ( int i = 0; i < count; ++i )
	{
		memset( items[i].stepScratch, 1 + i, sizeof( float ) * items[i].stepFloats * (size_t)chunk );
		memset( items[i].scratch, 1 + i, sizeof( float ) * ( CARRIED_FLOATS + (size_t)chunk ) );
	}
	for ( int i = 0; i < count; ++i )
		if ( *(char*)items[i].stepScratch != 1 + i || ( (char*)( items[i].scratch + CARRIED_FLOATS + chunk ) )[-1] != 1 + i )
			return -1;
	s_chunk = chunk;
	s_launches += 1;
	return cudaGetLastError();
}

static int fail( const char* what, int a, int b )
{
	printf( "failed: %s (%d, %d)\n", what, a, b );
	return 1;
}

int main( void )
{
	enum { STEPS = 120 };
	b2WorldId ids[2] = { { 0, 0 }, { 1, 0 } };
	b2gStepConst sc;
	memset( &sc, 0, sizeof( sc ) );
	sc.subSteps = 4;
	s_limit = (size_t)1 << 40;
	for ( int i = 0; i < 2; ++i )
	{
		gWorld* w = s_worlds + i;
		w->bodyIds.next = 3;
		w->shapeIds.next = 1;
		w->shapes = &s_shape;
		b2World_BeginTape( ids[i], STEPS );
		for ( int k = 0; k < STEPS; ++k )
			gtape_record( w, NULL, &sc, 0 );
		if ( b2World_GetTapeSteps( ids[i] ) != STEPS )
			return fail( "recording", i, 0 );
	}
	const size_t tapes = s_used;
	float final[2 * 6 * 3] = { 0 }, initial[2 * 6 * 3];
	const size_t step = 4u * 2u * STEP_FLOATS;
	/* memory for so many steps beside the tapes and the call's small buffers */
	static const int room[] = { 0, 1, 7, 31, 59, 60, 300 };
	for ( unsigned k = 0; k < sizeof( room ) / sizeof( room[0] ); ++k )
	{
		s_launches = 0;
		s_limit = tapes + 400000u + step * (size_t)room[k];
		int rc = b2World_StepBackwardBatch( ids, 2, 3, 1, final, initial, NULL );
		if ( room[k] == 0 ? rc != -1 || s_launches != 0 : rc != 0 || s_launches != 1 )
			return fail( "return code", room[k], rc );
		if ( room[k] > 0 && ( s_chunk > room[k] || ( 2 * s_chunk < STEPS && 2 * s_chunk + 1 < room[k] ) ) )
			return fail( "steps at a time", room[k], s_chunk );
	}
	if ( s_used <= tapes )
		return fail( "nothing is kept between calls", 0, 0 );
	b2World_BeginTape( ids[0], 0 );
	if ( s_used < tapes / 2 + step )
		return fail( "memory given back while a world has a tape", 0, 0 );
	b2World_BeginTape( ids[1], 0 );
	if ( s_used != 0 )
		return fail( "bytes kept after the last tape", (int)s_used, 0 );
	printf( "ok\n" );
	return 0;
}
