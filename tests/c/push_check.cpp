/*
 * push_check.cpp -- host model of the pushed body copies (box2c_gb300/csrc/b2g_push.h): CTAs
 * that sweep over coloured constraints, each with copies of the bodies its constraints
 * touch, an update of a body travelling as a message that completes on the receiver's
 * mbarrier of that sweep.  Messages arrive in any order and CTAs lag as they please; the
 * mbarriers count as the hardware's do.
 *
 * Checked on seeded random sets, some bodies of which are not integrated: every wait
 * ends, no transaction counts into a phase before its own, and every update starts from
 * the one before it.  Prints "ok" or the first failure.
 */
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
	/* then a restitution stage */
	TOTAL = SUBSTEPS * SWEEPS + COLORS,
	BARS = SWEEPS + COLORS,
};

enum Word
{
	VELOCITY,
	POSITION,
};

struct Constraint
{
	int cta, color, body[2];
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
};

struct Model
{
	const Set* set;
	bool forward; /* owners send the bodies they do not integrate as well */
	Bar bar[CTAS][BARS];
	int sweep[CTAS], armed[CTAS];
	std::vector<std::vector<int>> slot[2]; /* [word][cta][body]: the version held */
	std::vector<Message> flight;
	const char* fault = nullptr;
};

/* What sweep i is: its stage (-1 integrate, -2 positions, 0 to 3) and colour, and the
 * mbarrier it completes on. */
static void decode( int i, int* stage, int* color, int* bar, int* phase )
{
	*phase = i / SWEEPS;
	int k = i % SWEEPS;
	if ( i >= SUBSTEPS * SWEEPS )
	{
		*stage = 3;
		*color = i - SUBSTEPS * SWEEPS;
		*bar = SWEEPS + *color;
		*phase = 0;
		return;
	}
	*bar = k;
	*color = 0;
	if ( k == 0 )
		*stage = -1;
	else if ( k == 1 + 2 * COLORS )
		*stage = -2;
	else
	{
		k -= k > 2 * COLORS ? 2 : 1;
		*stage = k / COLORS;
		*color = k % COLORS;
	}
}

static bool moves( const Set& s, const Constraint& r, int b, int color ) { return r.color == color && ( r.body[0] == b || r.body[1] == b ); }

/* The CTA that updates body b's velocity in sweep i, or -1. */
static int updater( const Model& m, int b, int i )
{
	const Set& s = *m.set;
	int stage, color, bar, phase;
	decode( i, &stage, &color, &bar, &phase );
	if ( stage == -1 )
		return s.listed[b] || m.forward ? s.owner[b] : -1;
	for ( const Constraint& r : s.rows )
		if ( stage >= 0 && moves( s, r, b, color ) )
			return r.cta;
	return -1;
}

/* The CTA that updates its position, or -1. */
static int mover( const Model& m, int b, int i )
{
	int stage, color, bar, phase;
	decode( i, &stage, &color, &bar, &phase );
	return stage == -2 && ( m.set->listed[b] || m.forward ) ? m.set->owner[b] : -1;
}

/* The CTAs that the updater of sweep i sends the word of body b to. */
static unsigned receivers( const Model& m, int b, int i, Word word )
{
	const Set& s = *m.set;
	int stage, color, bar, phase;
	decode( i, &stage, &color, &bar, &phase );
	int from = word == VELOCITY ? updater( m, b, i ) : mover( m, b, i );
	if ( from < 0 )
		return 0;
	return s.holders[b] & ~( 1u << from );
}

static int version_before( const Model& m, int b, int i, Word word )
{
	int v = 0;
	for ( int k = 0; k < i; ++k )
		v += ( word == POSITION ? mover( m, b, k ) : updater( m, b, k ) ) >= 0;
	return v;
}

static int expected( const Model& m, int cta, int i )
{
	int n = 0;
	for ( int b = 0; b < m.set->bodies; ++b )
		for ( Word w : { VELOCITY, POSITION } )
			n += ( receivers( m, b, i, w ) >> cta ) & 1;
	return n;
}

/* CTA's own work of sweep i: it arms the sweep's mbarrier, updates and sends. */
static void begin_sweep( Model& m, int cta )
{
	const Set& s = *m.set;
	const int i = m.sweep[cta];
	int stage, color, bar, phase;
	decode( i, &stage, &color, &bar, &phase );
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
			int from = w == VELOCITY ? updater( m, b, i ) : mover( m, b, i );
			if ( from != cta )
				continue;
			int v = version_before( m, b, i, VELOCITY );
			if ( m.slot[VELOCITY][cta][b] != v && ( w == VELOCITY || s.listed[b] ) )
				m.fault = "an update starts from an older one";
			if ( stage >= 1 && stage <= 2 && m.slot[POSITION][cta][b] != version_before( m, b, i, POSITION ) )
				m.fault = "a constraint reads an older position";
			v = version_before( m, b, i, w ) + 1;
			m.slot[w][cta][b] = v;
			unsigned to = receivers( m, b, i, w );
			for ( int t = 0; t < CTAS; ++t )
				if ( ( to >> t ) & 1 )
					m.flight.push_back( { t, b, i, v, w } );
		}
}

static void deliver( Model& m, size_t k )
{
	Message g = m.flight[k];
	m.flight.erase( m.flight.begin() + (long)k );
	int stage, color, bar, phase;
	decode( g.sweep, &stage, &color, &bar, &phase );
	Bar& B = m.bar[g.to][bar];
	if ( B.phase != phase )
		m.fault = "a transaction counts into a phase before its own";
	m.slot[g.word][g.to][g.body] = g.version;
	B.tx -= 1;
	B.settle();
}

/* Runs the set under one schedule: CTA `lag` moves seldom.  Messages of one sweep may
 * overtake one another, later ones none of the same body. */
static const char* run( const Set& s, bool forward, int lag )
{
	Model m;
	m.set = &s;
	m.forward = forward;
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
			return nullptr;
		if ( m.flight.empty() == false && rnd( 3 ) != 0 )
		{
			int k = rnd( (int)m.flight.size() );
			for ( int j = 0; j < k; ++j )
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
		int stage, color, bar, phase;
		decode( m.sweep[c], &stage, &color, &bar, &phase );
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
		Constraint r = { rnd( CTAS ), 1 + rnd( COLORS - 1 ), { rnd( s.bodies ), rnd( s.bodies ) } };
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
	for ( int b = 0; b < s.bodies; ++b )
		s.holders[b] = 1u << s.owner[b];
	for ( const Constraint& r : s.rows )
		for ( int b : r.body )
			if ( b >= 0 )
				s.holders[b] |= 1u << r.cta;
	return s;
}

int main()
{
	int caught = 0;
	for ( int k = 0; k < 800; ++k )
	{
		Set s = make_set();
		int lag = rnd( CTAS + 1 );
		const char* fault = run( s, true, lag );
		if ( fault )
		{
			printf( "failed: %s (set %d, %d bodies)\n", fault, k, s.bodies );
			return 1;
		}
		/* with owners silent about the bodies they do not integrate, a CTA runs ahead of one */
		fault = run( s, false, lag );
		caught += fault != nullptr && strstr( fault, "before its own" ) != nullptr;
	}
	if ( caught < 8 )
	{
		printf( "failed: the planted mistake was met %d times\n", caught );
		return 1;
	}
	printf( "ok: 800 sets, planted mistake met %d times\n", caught );
	return 0;
}
