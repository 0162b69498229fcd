/*
 * b2g_space.h -- what the CTAs of a resident contact solve hold in shared memory
 * (resident.cu, fused.cu): plain arithmetic, for the host alone.
 */
#pragma once

#include "b2g_types.h"

#include <stddef.h>

/* dynamic shared memory per CTA, leaving 1 KB of the 227 KB opt-in limit for statics */
#define RES_SMEM_MAX ( 226 * 1024 )
/* overflow rows of a set that keeps its bodies in a cache of CTA 0 */
#define RES_OVERFLOW_MAX 512
/* bytes of one row, and of one body slot: two state float4, the velocity terms (float4 and
 * float), flags and an entry of the awake list */
#define RES_ROW_BYTES 144
#define RES_BODY_BYTES 60

#ifdef __CUDACC__
#define RES_SPACE_FN static inline __host__ __device__
#else
#define RES_SPACE_FN static inline
#endif

/* Overflow cache of R rows and J joints (ResOverflow). */
RES_SPACE_FN size_t res_overflow_bytes( int R, int J )
{
	size_t E = 2u * (size_t)( R + J );
	return 16u * ( (size_t)R + 2u * E ) + 4u * ( 3u * E + 2u * (size_t)J );
}

/* Row slots of the fullest CTA: every colour splits into shares that differ by one, CTA
 * 0 also holds the overflow rows. */
static inline int res_row_cap( const int* cs, int ctas )
{
	int cap = cs[B2G_COLORS] - cs[B2G_OVERFLOW];
	for ( int c = 0; c < B2G_OVERFLOW; ++c )
		cap += ( cs[c + 1] - cs[c] + ctas - 1 ) / ctas;
	return cap > 0 ? cap : 1;
}

/* The body slots of a CTA when the set's rows fit the shared memory of `ctas` CTAs with as
 * many bodies as it lists and one for every two rows (body indices are the caller's: the
 * kernel copes with more, at L2); 0 when they do not.  The slots take what the rows and
 * CTA 0's overflow cache leave, so they are never fewer than a CTA's share of the list. */
static inline int res_body_cap( const int* cs, int listed, int ctas )
{
	const int ovRows = cs[B2G_COLORS] - cs[B2G_OVERFLOW];
	int want = listed > cs[B2G_COLORS] / 2 ? listed : cs[B2G_COLORS] / 2;
	want = ( want + ctas - 1 ) / ctas + 1;
	const size_t rows = RES_ROW_BYTES * (size_t)res_row_cap( cs, ctas );
	const size_t tail = ctas > 1 && ovRows > 0 && ovRows <= RES_OVERFLOW_MAX ? res_overflow_bytes( ovRows, 0 ) + 16 : 0;
	if ( rows + RES_BODY_BYTES * (size_t)want + tail > RES_SMEM_MAX )
		return 0;
	const int most = (int)( ( RES_SMEM_MAX - rows - tail ) / RES_BODY_BYTES );
	return most < 4 * want ? most : 4 * want;
}
