/*
 * push_check.cpp -- host model of the pushed body copies (box2c_gb300/csrc/b2g_push.h): CTAs
 * that sweep over coloured constraints, each with copies of the bodies its constraints
 * touch, an update of a body travelling as a message that completes on the receiver's
 * mbarrier of that sweep, to the CTA that box2c_gb300/csrc/b2g_chain.h names.  Messages
 * arrive in any order, CTAs lag as they please, and the mbarriers count as the hardware's
 * do.
 *
 * Checked on seeded random sets, some bodies of which are not integrated: every wait
 * ends, no transaction counts into a phase before its own, every update starts from the
 * one before it, and the owner ends with the last one.  Prints "ok" or the first failure.
 */
#include "b2g_chain.h"

#include <algorithm>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>
#include <vector>

static unsigned long long s_state = 2463534242ull;
static int rnd( int n )
{
	s_state = s_state * 6364136223846793005ull + 1442695040888963407ull;
	return (int)( ( s_state >> 33 ) % (unsigned long long)n );
}

enum
{
	CTAS = 6,
	COLORS = 5, /* colour 0 is the overflow set, which CTA 0 solves first in every stage */
	SUBSTEPS = 4,
	/* sweeps of a substep: integrate, warm start, solve, positions, relax */
	SWEEPS = 2 + 3 * COLORS,
	/* then the start of restitution and its stage */
	TOTAL = SUBSTEPS * SWEEPS + 1 + COLORS,
	BARS = SWEEPS + 1 + COLORS,
};

/* How updates travel: to the next updater, or to all copies; with the latter, owners may
 * send nothing of the bodies that they do not integrate. */
enum Policy
{
	CHAIN,
	ALL,
	ALL_LISTED,
};

enum Word
{
	VELOCITY,
	POSITION,
};

struct Constraint
{
	int cta, color, joint, body[2];
};

/* An mbarrier of arrival count 1. */
struct Bar
{
	int phase = 0, pending = 1, tx = 0;
	void settle()
	{
		if ( pending == 0 && tx == 0 )
		{
			phase += 1;
			pending = 1;
		}
	}
};

struct Message
{
	int to, body, sweep, version;
	Word word;
};

struct Set
{
	int bodies;
	std::vector<int> owner, listed;
	std::vector<Constraint> rows;
	std::vector<unsigned> holders; /* CTAs with a copy, the owner among them */
	std::vector<b2gChain> chain;
};

struct Model
{
	const Set* set;
	Policy policy;
	Bar bar[CTAS][BARS];
	int sweep[CTAS], armed[CTAS];
	std::vector<std::vector<int>> slot[2]; /* [word][cta][body]: the version held */
	std::vector<Message> flight;
	const char* fault = nullptr;
};

enum Stage
{
	WARM,
	SOLVE,
	RELAX,
	RESTITUTION,
	INTEGRATE,
	POSITIONS,
	RESTITUTION_START,
};

/* What sweep i is: its stage and colour, and the mbarrier it completes on. */
static Stage decode( int i, int* color, int* bar, int* phase )
{
	*phase = i / SWEEPS;
	*color = 0;
	int k = i % SWEEPS;
	if ( i >= SUBSTEPS * SWEEPS )
	{
		k = i - SUBSTEPS * SWEEPS;
		*phase = 0;
		*bar = SWEEPS + k;
		*color = k > 0 ? k - 1 : 0;
		return k == 0 ? RESTITUTION_START : RESTITUTION;
	}
	*bar = k;
	if ( k == 0 )
		return INTEGRATE;
	if ( k == 1 + 2 * COLORS )
		return POSITIONS;
	k -= k > 2 * COLORS ? 2 : 1;
	*color = k % COLORS;
	return (Stage)( k / COLORS );
}

static bool sent_by_owner( const Model& m, int b ) { return m.set->listed[b] || m.policy != ALL_LISTED; }

/* The CTA that updates a word of body b in sweep i, or -1. */
static int updater( const Model& m, int b, int i, Word word )
{
	int color, bar, phase;
	const Stage stage = decode( i, &color, &bar, &phase );
	if ( stage == ( word == VELOCITY ? INTEGRATE : POSITIONS ) )
		return sent_by_owner( m, b ) ? m.set->owner[b] : -1;
	if ( word == POSITION || stage > RESTITUTION )
		return -1;
	for ( const Constraint& r : m.set->rows )
		if ( r.color == color && ( r.body[0] == b || r.body[1] == b ) && ( r.joint == 0 || stage != RESTITUTION ) )
			return r.cta;
	return -1;
}

/* The CTA that sends a word in sweep i, or -1, and the CTAs it goes to. */
static int sender( const Model& m, int b, int i, Word word, unsigned* to )
{
	const Set& s = *m.set;
	int color, bar, phase;
	const Stage stage = decode( i, &color, &bar, &phase );
	int from = updater( m, b, i, word );
	*to = 0;
	if ( m.policy != CHAIN || word == POSITION )
	{
		if ( from >= 0 )
			*to = s.holders[b] & ~( 1u << from );
		return from;
	}
	if ( stage == POSITIONS || stage == RESTITUTION_START )
		from = s.owner[b];
	if ( from < 0 )
		return -1;
	int t = b2g_chain_next( s.chain[b], stage > RESTITUTION ? -1 : color, stage == WARM, stage == RESTITUTION || stage == RESTITUTION_START,
							s.owner[b] );
	*to = 1u << t & ~( 1u << from );
	return from;
}

static int version_before( const Model& m, int b, int i, Word word )
{
	int v = 0;
	for ( int k = 0; k < i; ++k )
		v += updater( m, b, k, word ) >= 0;
	return v;
}

static int expected( const Model& m, int cta, int i )
{
	int n = 0;
	unsigned to;
	for ( int b = 0; b < m.set->bodies; ++b )
		for ( Word w : { VELOCITY, POSITION } )
		{
			sender( m, b, i, w, &to );
			n += ( to >> cta ) & 1;
		}
	return n;
}

/* CTA's own work of sweep i: it arms the sweep's mbarrier, updates and sends. */
static void begin_sweep( Model& m, int cta )
{
	const Set& s = *m.set;
	const int i = m.sweep[cta];
	int color, bar, phase;
	const Stage stage = decode( i, &color, &bar, &phase );
	int n = expected( m, cta, i );
	if ( n > 0 )
	{
		Bar& B = m.bar[cta][bar];
		if ( B.phase != phase )
			m.fault = "a sweep's mbarrier is in another phase";
		B.pending -= 1;
		B.tx += n;
		B.settle();
	}
	m.armed[cta] = 1;
	for ( int b = 0; b < s.bodies; ++b )
		for ( Word w : { VELOCITY, POSITION } )
		{
			unsigned to;
			if ( sender( m, b, i, w, &to ) != cta )
				continue;
			const bool update = updater( m, b, i, w ) == cta;
			if ( ( update || to ) && m.slot[VELOCITY][cta][b] != version_before( m, b, i, VELOCITY ) )
				m.fault = "an update starts from an older one";
			if ( ( stage == SOLVE || stage == RELAX ) && m.slot[POSITION][cta][b] != version_before( m, b, i, POSITION ) )
				m.fault = "a constraint reads an older position";
			const int v = version_before( m, b, i, w ) + update;
			/* a velocity that goes to the next updater is not kept */
			if ( m.policy != CHAIN || w == POSITION || to == 0 )
				m.slot[w][cta][b] = v;
			for ( int t = 0; t < CTAS; ++t )
				if ( ( to >> t ) & 1 )
					m.flight.push_back( { t, b, i, v, w } );
		}
}

static void deliver( Model& m, size_t k )
{
	Message g = m.flight[k];
	m.flight.erase( m.flight.begin() + (long)k );
	int color, bar, phase;
	decode( g.sweep, &color, &bar, &phase );
	Bar& B = m.bar[g.to][bar];
	if ( B.phase != phase )
		m.fault = "a transaction counts into a phase before its own";
	m.slot[g.word][g.to][g.body] = g.version;
	B.tx -= 1;
	B.settle();
}

/* Runs the set under one schedule: CTA `lag` moves seldom.  A message may overtake any
 * other, or with `ordered` none of the same copy. */
static const char* run( const Set& s, Policy policy, int lag, bool ordered )
{
	Model m;
	m.set = &s;
	m.policy = policy;
	for ( int w = 0; w < 2; ++w )
		m.slot[w].assign( CTAS, std::vector<int>( (size_t)s.bodies, 0 ) );
	for ( int c = 0; c < CTAS; ++c )
		m.sweep[c] = m.armed[c] = 0;
	for ( int idle = 0; idle < 200000; ++idle )
	{
		int left = 0;
		for ( int c = 0; c < CTAS; ++c )
			left += m.sweep[c] < TOTAL;
		if ( m.fault )
			return m.fault;
		if ( left == 0 && m.flight.empty() )
		{
			for ( int b = 0; b < s.bodies; ++b )
				if ( m.slot[VELOCITY][s.owner[b]][b] != version_before( m, b, TOTAL, VELOCITY ) )
					return "an owner ends with an older velocity";
			return nullptr;
		}
		if ( m.flight.empty() == false && rnd( 3 ) != 0 )
		{
			int k = rnd( (int)m.flight.size() );
			for ( int j = 0; j < k && ordered; ++j )
				if ( m.flight[j].to == m.flight[k].to && m.flight[j].body == m.flight[k].body )
				{
					k = j;
					break;
				}
			deliver( m, (size_t)k );
			idle = 0;
			continue;
		}
		int c = rnd( CTAS );
		if ( m.sweep[c] == TOTAL || ( c == lag && rnd( 40 ) != 0 ) )
			continue;
		if ( m.armed[c] == 0 )
		{
			begin_sweep( m, c );
			idle = 0;
			continue;
		}
		int color, bar, phase;
		decode( m.sweep[c], &color, &bar, &phase );
		if ( expected( m, c, m.sweep[c] ) > 0 && m.bar[c][bar].phase == phase )
			continue;
		m.sweep[c] += 1;
		m.armed[c] = 0;
		idle = 0;
	}
	return "a wait does not end";
}

static Set make_set()
{
	Set s;
	s.bodies = 2 + rnd( 14 );
	for ( int b = 0; b < s.bodies; ++b )
	{
		s.owner.push_back( rnd( CTAS ) );
		s.listed.push_back( rnd( 4 ) != 0 );
	}
	int want = 1 + rnd( 3 * s.bodies );
	for ( int k = 0; k < want; ++k )
	{
		Constraint r = { rnd( CTAS ), 1 + rnd( COLORS - 1 ), rnd( 5 ) == 0, { rnd( s.bodies ), rnd( s.bodies ) } };
		if ( rnd( 8 ) == 0 )
			r.body[1] = -1;
		if ( r.body[0] == r.body[1] )
			continue;
		bool taken = false;
		for ( const Constraint& q : s.rows )
			for ( int e = 0; e < 2; ++e )
				taken = taken || ( q.color == r.color && r.body[e] >= 0 && ( q.body[0] == r.body[e] || q.body[1] == r.body[e] ) );
		/* one overflow constraint of a body here, as the set is one update of it */
		if ( taken )
		{
			r.color = 0;
			r.cta = 0;
			for ( const Constraint& q : s.rows )
				for ( int e = 0; e < 2; ++e )
					if ( q.color == 0 && r.body[e] >= 0 && ( q.body[0] == r.body[e] || q.body[1] == r.body[e] ) )
						r.cta = -1;
			if ( r.cta < 0 || rnd( 3 ) == 0 )
				continue;
		}
		s.rows.push_back( r );
	}
	s.holders.assign( (size_t)s.bodies, 0u );
	s.chain.assign( (size_t)s.bodies, b2gChain{ 0u, { 0u, 0u } } );
	for ( int b = 0; b < s.bodies; ++b )
		s.holders[b] = 1u << s.owner[b];
	for ( const Constraint& r : s.rows )
		for ( int b : r.body )
			if ( b >= 0 )
			{
				s.holders[b] |= 1u << r.cta;
				s.chain[b].who |= 1u << ( r.color + ( r.joint ? 16 : 0 ) );
				s.chain[b].cta[r.color >> 3] |= (unsigned)r.cta << ( 4 * ( r.color & 7 ) );
			}
	return s;
}

/* b2g_chain_next over all 12 places, CTAs and subsets against a walk of the stages. */
static const char* check_chain( void )
{
	for ( int n = 0; n < 20000; ++n )
	{
		b2gChain c = { 0u, { 0u, 0u } };
		int cta[B2G_CHAIN_PLACES], kind[B2G_CHAIN_PLACES];
		const int owner = rnd( 16 );
		for ( int p = 0; p < B2G_CHAIN_PLACES; ++p )
		{
			kind[p] = rnd( 3 ) == 0 ? 1 + rnd( 2 ) : 0; /* 1 a row, 2 a joint */
			cta[p] = p == 0 ? 0 : rnd( 16 );
			if ( kind[p] )
			{
				c.who |= 1u << ( p + ( kind[p] == 2 ? 16 : 0 ) );
				c.cta[p >> 3] |= (unsigned)cta[p] << ( 4 * ( p & 7 ) );
			}
		}
		for ( int restitution = 0; restitution < 2; ++restitution )
			for ( int warm = 0; warm < 2 - restitution; ++warm )
				for ( int p = -1; p < B2G_CHAIN_PLACES; ++p )
				{
					int want = -1;
					for ( int lap = 0; lap < ( warm ? 2 : 1 ) && want < 0; ++lap )
						for ( int q = lap ? 0 : p + 1; q < B2G_CHAIN_PLACES && want < 0; ++q )
							want = kind[q] == 1 || ( kind[q] == 2 && restitution == 0 ) ? cta[q] : -1;
					want = want < 0 ? owner : want;
					if ( b2g_chain_next( c, p, warm, restitution, owner ) != want )
						return "the next CTA of a chain";
				}
	}
	return nullptr;
}

int main()
{
	const char* wrong = check_chain();
	if ( wrong )
	{
		printf( "failed: %s\n", wrong );
		return 1;
	}
	int ahead = 0, stale = 0;
	for ( int k = 0; k < 500; ++k )
	{
		Set s = make_set();
		int lag = rnd( CTAS + 1 );
		const char* fault = run( s, CHAIN, lag, false );
		if ( fault )
		{
			printf( "failed: %s (set %d, %d bodies)\n", fault, k, s.bodies );
			return 1;
		}
		/* updates sent to all copies overtake one another; with owners silent about the bodies
		 * that they do not integrate, a CTA runs ahead of one even where they do not */
		fault = run( s, ALL, lag, false );
		stale += fault != nullptr && strstr( fault, "older" ) != nullptr;
		fault = run( s, ALL_LISTED, lag, true );
		ahead += fault != nullptr && strstr( fault, "before its own" ) != nullptr;
		if ( ( fault = run( s, ALL, lag, true ) ) != nullptr )
		{
			printf( "failed: %s with ordered messages (set %d)\n", fault, k );
			return 1;
		}
	}
	if ( ahead < 5 || stale < 5 )
	{
		printf( "failed: planted mistakes were met %d and %d times\n", ahead, stale );
		return 1;
	}
	printf( "ok: 500 sets, planted mistakes met %d and %d times\n", ahead, stale );
	return 0;
}
