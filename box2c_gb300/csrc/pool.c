/*
 * pool.c -- a small fork-join thread pool for the host side of batched steps: the
 * per-world host work of b2World_StepBatch is independent between worlds, and touching
 * thousands of separately allocated worlds is bound by memory latency, so it spreads
 * over the host's cores.
 *
 * gpool_for( count, grain, fn, ctx ) calls fn( begin, end, ctx ) over [0, count) in
 * chunks of `grain`, on the calling thread and the pool's workers, and returns when all
 * chunks are done.  One job runs at a time: gpool_for waits for the pool, gpool_try_for
 * returns false at once when the pool is busy (another thread's job, or a call from
 * inside a job) and the caller runs the range itself.  gpool_for must not nest.
 *
 * A batched step has five short jobs, microseconds of work each for a hundred worlds, so
 * what counts is what a job costs beside its work.  The caller waits only for workers
 * that are inside the job, never for one that still has to wake up, and a worker watches
 * for the next job for POOL_WATCH_US before it sleeps.  Waking every worker and waiting
 * for all of them took 30 to 60 us a job (96 worlds of 8 bodies: 293 us a step with it,
 * 142 without).
 */
#include "host.h"

#include <pthread.h>
#include <sched.h>
#include <stdatomic.h>
#include <stdlib.h>
#include <time.h>
#include <unistd.h>

#define POOL_MAX_THREADS 32
#define POOL_WATCH_US 100

typedef struct gPool
{
	pthread_t threads[POOL_MAX_THREADS];
	int workers;
	pthread_mutex_t lock; /* sleeping workers */
	pthread_cond_t wake;
	int sleeping;
	/* the open job's number, 0 when none is open: its fields do not change while it is
	 * open, nor while a worker that found it open is inside */
	atomic_ullong open;
	unsigned long long jobs;
	gTaskFn* fn;
	void* ctx;
	int count, grain;
	atomic_int next;
	atomic_int inside;
} gPool;

static gPool s_pool;
static pthread_once_t s_once = PTHREAD_ONCE_INIT;
static pthread_mutex_t s_job = PTHREAD_MUTEX_INITIALIZER; /* held while a job runs */

static void run_chunks( gPool* p )
{
	for ( ;; )
	{
		int begin = atomic_fetch_add( &p->next, p->grain );
		if ( begin >= p->count )
			break;
		int end = begin + p->grain < p->count ? begin + p->grain : p->count;
		p->fn( begin, end, p->ctx );
	}
}

static long long now_us( void )
{
	struct timespec t;
	clock_gettime( CLOCK_MONOTONIC, &t );
	return 1000000ll * t.tv_sec + t.tv_nsec / 1000;
}

static void* worker( void* arg )
{
	gPool* p = (gPool*)arg;
	unsigned long long seen = 0;
	for ( ;; )
	{
		/* watch for a job, then sleep until one is opened */
		unsigned long long job = atomic_load( &p->open );
		for ( long long until = now_us() + POOL_WATCH_US; job == 0 || job == seen; job = atomic_load( &p->open ) )
		{
			if ( now_us() < until )
			{
				sched_yield();
				continue;
			}
			pthread_mutex_lock( &p->lock );
			for ( job = atomic_load( &p->open ); job == 0 || job == seen; job = atomic_load( &p->open ) )
			{
				p->sleeping += 1;
				pthread_cond_wait( &p->wake, &p->lock );
				p->sleeping -= 1;
			}
			pthread_mutex_unlock( &p->lock );
			break;
		}
		/* enter it unless it has closed meanwhile */
		atomic_fetch_add( &p->inside, 1 );
		job = atomic_load( &p->open );
		if ( job != 0 && job != seen )
		{
			seen = job;
			run_chunks( p );
		}
		atomic_fetch_sub( &p->inside, 1 );
	}
	return NULL;
}

static void pool_start( void )
{
	gPool* p = &s_pool;
	pthread_mutex_init( &p->lock, NULL );
	pthread_cond_init( &p->wake, NULL );
	long cores = sysconf( _SC_NPROCESSORS_ONLN );
	int n = cores > 1 ? (int)cores - 1 : 0;
	n = n > POOL_MAX_THREADS ? POOL_MAX_THREADS : n;
	int started = 0;
	for ( int i = 0; i < n; ++i )
	{
		if ( pthread_create( p->threads + started, NULL, worker, p ) == 0 )
			started += 1;
	}
	p->workers = started;
}

int gpool_threads( void )
{
	pthread_once( &s_once, pool_start );
	return s_pool.workers + 1;
}

static void run_job( int count, int grain, gTaskFn* fn, void* ctx )
{
	gPool* p = &s_pool;
	p->fn = fn;
	p->ctx = ctx;
	p->count = count;
	p->grain = grain;
	atomic_store( &p->next, 0 );
	p->jobs += 1;
	atomic_store( &p->open, p->jobs );
	/* wake as many more as there are chunks for */
	int wanted = ( count + grain - 1 ) / grain - 1;
	wanted = wanted > p->workers ? p->workers : wanted;
	pthread_mutex_lock( &p->lock );
	int wakes = wanted - ( p->workers - p->sleeping );
	pthread_mutex_unlock( &p->lock );
	for ( int i = 0; i < wakes; ++i )
		pthread_cond_signal( &p->wake );
	run_chunks( p );
	/* no chunk is left to take: close, and wait for those that are being run */
	atomic_store( &p->open, 0 );
	while ( atomic_load( &p->inside ) > 0 )
		sched_yield();
}

void gpool_for( int count, int grain, gTaskFn* fn, void* ctx )
{
	if ( count <= 0 )
		return;
	grain = grain < 1 ? 1 : grain;
	pthread_once( &s_once, pool_start );
	if ( s_pool.workers == 0 || count <= grain )
	{
		fn( 0, count, ctx );
		return;
	}
	pthread_mutex_lock( &s_job );
	run_job( count, grain, fn, ctx );
	pthread_mutex_unlock( &s_job );
}

bool gpool_try_for( int count, int grain, gTaskFn* fn, void* ctx )
{
	if ( count <= 0 )
		return true;
	grain = grain < 1 ? 1 : grain;
	pthread_once( &s_once, pool_start );
	if ( s_pool.workers == 0 || count <= grain )
		return false;
	if ( pthread_mutex_trylock( &s_job ) != 0 )
		return false;
	run_job( count, grain, fn, ctx );
	pthread_mutex_unlock( &s_job );
	return true;
}
