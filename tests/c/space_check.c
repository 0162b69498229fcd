/*
 * space_check.c -- what the CTAs of a resident contact solve hold (b2g_space.h), over every
 * number of listed bodies up to past the largest that fits, for one CTA and a cluster, sets
 * with and without overflow rows: where a set is taken, a CTA has a slot for each of its
 * share of the bodies (0 to listed - 1, or the list itself), and rows, slots and overflow
 * cache fit; a set that would fit is taken.  Prints "ok" or the first failure.
 */
#include "b2g_device.h"
#include "b2g_space.h"

#include <stdio.h>

static int check( const int* cs, int listed, int ctas, int* taken )
{
	const int ovRows = cs[B2G_COLORS] - cs[B2G_OVERFLOW], share = ( listed + ctas - 1 ) / ctas;
	const int cap = res_body_cap( cs, listed, ctas );
	size_t bytes = 144u * (size_t)res_row_cap( cs, ctas );
	const int cache = ctas > 1 && ovRows > 0 && ovRows <= RES_OVERFLOW_MAX;
	const int half = ( cs[B2G_COLORS] / 2 + ctas - 1 ) / ctas, most = share > half ? share : half;
	*taken = cap > 0;
	if ( cap == 0 )
		return bytes + 60u * (size_t)( most + 1 ) + ( cache ? res_overflow_bytes( ovRows, 0 ) + 16u : 0u ) <= RES_SMEM_MAX;
	bytes += 60u * (size_t)cap;
	if ( cache )
		bytes = ( bytes + 15 ) / 16 * 16 + res_overflow_bytes( ovRows, 0 );
	return cap < most || bytes > RES_SMEM_MAX;
}

int main( void )
{
	static const int sets[][2] = { { 0, 0 }, { 1, 0 }, { 1001, 0 }, { 1014, 0 }, { 1201, 0 }, { 1299, 0 }, { 1300, 40 },
								   { 1599, 0 }, { 3000, 17 }, { 15000, 0 }, { 15654, 0 }, { 16000, 511 }, { 20000, 600 }, { 25000, 0 } };
	for ( int ctas = 1; ctas <= B2G_FUSED_CTAS; ctas += B2G_FUSED_CTAS - 1 )
		for ( unsigned k = 0; k < sizeof( sets ) / sizeof( sets[0] ); ++k )
			for ( int colours = 1; colours <= 11; colours += 5 )
			{
				int cs[B2G_COLORS + 1] = { 0 };
				const int rest = sets[k][0] - sets[k][1];
				for ( int c = 0; c < B2G_OVERFLOW; ++c )
					cs[c + 1] = c < colours ? (int)( (long long)rest * ( c + 1 ) / colours ) : rest;
				cs[B2G_COLORS] = sets[k][0];
				int was = 1, taken = 0;
				for ( int listed = 0; listed < 4000 * ctas; ++listed )
				{
					if ( check( cs, listed, ctas, &taken ) || ( taken && was == 0 ) )
					{
						printf( "failed: %d contacts (%d overflow) in %d colours, %d bodies, %d CTAs\n", sets[k][0], sets[k][1], colours, listed, ctas );
						return 1;
					}
					was = taken;
				}
				if ( taken )
				{
					printf( "failed: no edge for %d contacts\n", sets[k][0] );
					return 1;
				}
			}
	printf( "ok\n" );
	return 0;
}
