/*
 * adjoint.cu -- reverse-mode gradient of recorded steps (b2World_StepBackward).
 *
 * Forward: while a world's tape is active, every step records its solver inputs before
 * the solver stage runs (k_tape_record): body states at the step start and the
 * coloured rows with the manifolds the narrowphase produced (warm-start impulses
 * included).
 *
 * Backward, in chunks of steps from the last to the first:
 *   k_adjoint_replay   one warp per world and step, all steps of a chunk at once: a step
 *                      depends only on its record.  It is replayed forward -- the same
 *                      b2g_solve.h arithmetic in the same order, so the replay is
 *                      bit-identical -- keeping body snapshots and, for every row and
 *                      phase, the velocities before each of its impulses; the contact
 *                      geometry is recomputed with dual numbers (b2g_dual.h) for its
 *                      Jacobian.
 *   k_adjoint_reverse  one warp per world, the chunk's steps in reverse: finalisation,
 *                      restitution colours in reverse order, and per substep in reverse:
 *                      relax colours reversed, position integration, solve colours
 *                      reversed, warm-start colours reversed, velocity integration; then
 *                      the row preparation and the narrowphase Jacobian.  A step's
 *                      replay comes into shared memory by a bulk copy while the step
 *                      after it is differentiated.
 *   k_adjoint_friction one thread per shape: the friction gradient's sums, in step and
 *                      row order.
 * Only the reverse pass is a chain over the steps, and it is bound by that chain: about
 * 18 us a step of some 70 dependent sweeps.  96 worlds of 8 boxes and 120 steps, one warp
 * a world doing replay, Jacobians and reverse in turn before: 10.9 ms a call; now 3.2 ms
 * (replay 0.68, reverse 2.13, friction 0.03).  Replaying the next chunk on a second
 * stream beside the reverse pass took 3.6 ms: the two share the SMs' issue slots.
 *
 * Within a colour no two rows share a body, so a colour's row adjoints run in parallel
 * lanes without conflicts.  The adjoint of the warm-start impulses goes to the previous
 * step's stored impulses through the narrowphase's feature-id matching (reference
 * src/contact.c:555-568).
 *
 * Differentiated: body centres, angles, linear and angular velocities, and contact
 * friction (mixed per shape as sqrt(muA * muB), reference src/contact.c:42-45).  The
 * discrete choices of a step (pairs, colours, manifold features, active clamps) are
 * those of the recorded forward step.  Polygon, capsule, segment and circle shapes, and
 * rows in the graph colours and in the overflow colour; joints and chain links are
 * reported as unsupported.
 *
 * Reference arithmetic being differentiated: src/solver.c:34-93, :146-163, :205-223;
 * src/contact_solver.c:597-1293; src/manifold.c:276-700.
 */
#include "b2g_dual.h"
#include "b2g_stages.h"

#include <cuda_runtime.h>

/* ------------------------------------------------------------------ recording */
__global__ void k_tape_record( b2gDevWorld W, float4* bodies, int bodyCount, b2gTapeRow* rows, int rowCount )
{
	tape_record_one( W, bodies, bodyCount, rows, rowCount, blockIdx.x * blockDim.x + threadIdx.x );
}

extern "C" int b2gd_tape_record( b2gDevWorld* w, void* bodyDst, int bodies, void* rowDst, int rows )
{
	int n = bodies > rows ? bodies : rows;
	if ( n <= 0 )
		return 0;
	k_tape_record<<<( n + 255 ) / 256, 256, 0, (cudaStream_t)w->stream>>>( *w, (float4*)bodyDst, bodies, (b2gTapeRow*)rowDst, rows );
	return (int)cudaGetLastError();
}

/* ------------------------------------------------------------------ scratch layout */
#define ADJ_BODY 12
#define ADJ_STATE 8
#define ADJ_START 9
#define ADJ_TERMS 5
#define ADJ_SNAP 8
#define ADJ_RADJ 24
#define ADJ_JAC 72
#define ADJ_MAX_SUBSTEPS 16
/* what the reverse pass reads of a row: bodies, count, normal, friction, restitution,
 * masses, anchors, coefficients and the link to the previous step's row; of its phases: the impulses and the velocities of
 * both bodies before each impulse (none for a warm start, four for solve and relax, two
 * for restitution) */
#define ADJ_ROW 28
#define ADJ_WARM 4
#define ADJ_SOLVE 28
#define ADJ_REST 16

/* One step's replay, as the reverse pass reads it: field f of row k at [f * Rs + k], of
 * body b at [f * Ns + b], offsets in floats; then the replay's own working arrays. */
struct AdjStep
{
	int Rs, Ns, S;
	size_t rows, phase, jac, snap, start, terms;
	size_t copy; /* floats of the parts above */
	size_t work, state, total;

	__host__ __device__ size_t warm( int sub ) const { return phase + (size_t)sub * ( ADJ_WARM + 2 * ADJ_SOLVE ) * Rs; }
	__host__ __device__ size_t solve( int sub, int relax ) const { return warm( sub ) + (size_t)( ADJ_WARM + ADJ_SOLVE * relax ) * Rs; }
	__host__ __device__ size_t rest() const { return warm( S ); }
};

static __host__ __device__ AdjStep adj_step( int N, int R, int S )
{
	AdjStep l;
	l.Rs = ( R + 3 ) & ~3;
	l.Ns = ( N + 3 ) & ~3;
	l.S = S;
	size_t o = 0, Rs = (size_t)l.Rs, Ns = (size_t)l.Ns;
	l.rows = o;
	o += ADJ_ROW * Rs;
	l.phase = o;
	o += ( (size_t)S * ( ADJ_WARM + 2 * ADJ_SOLVE ) + ADJ_REST ) * Rs;
	l.jac = o;
	o += ADJ_JAC * Rs;
	l.snap = o;
	o += (size_t)( 2 * S + 1 ) * ADJ_SNAP * Ns;
	l.start = o;
	o += ADJ_START * Ns;
	l.terms = o;
	o += ADJ_TERMS * Ns;
	l.copy = o;
	l.work = o;
	o += sizeof( Row ) / 4 * Rs;
	l.state = o;
	o += ADJ_STATE * Ns;
	l.total = o;
	return l;
}

/* What a world carries from step to step: body adjoints, rotation and local centre at the
 * last differentiated step's start (4 per body), impulse adjoints of the step to come and
 * the one before it (4 per row each), friction adjoints of a chunk's rows. */
struct AdjWorld
{
	float* bodyAdj;
	float* pose;
	float* lam;
	float* mu;
};

static __host__ __device__ size_t adj_world( AdjWorld* L, float* base, int N, int R, int chunk )
{
	size_t o = 0;
	auto take = [&]( size_t n ) {
		float* p = base ? base + o : nullptr;
		o += ( n + 3 ) & ~(size_t)3;
		return p;
	};
	AdjWorld l;
	l.bodyAdj = take( (size_t)N * ADJ_BODY );
	l.pose = take( (size_t)N * 4 );
	l.lam = take( (size_t)R * 8 );
	l.mu = take( (size_t)R * chunk );
	if ( L )
		*L = l;
	return o;
}

static int at_least_one( int v ) { return v < 1 ? 1 : v; }

/* Scratch floats of one world: carried from step to step, and of one step's replay. */
extern "C" size_t b2gd_adjoint_scratch( int bodies, int maxRows, int chunk )
{
	AdjStep l = adj_step( bodies, at_least_one( maxRows ), 1 );
	return adj_world( nullptr, nullptr, l.Ns, l.Rs, chunk );
}

/* with the table of the previous step's rows by contact id */
extern "C" size_t b2gd_adjoint_step_scratch( int bodies, int maxRows, int contactCap, int subSteps )
{
	return adj_step( bodies, at_least_one( maxRows ), subSteps ).total + ( ( (size_t)at_least_one( contactCap ) + 3 ) & ~(size_t)3 );
}

/* ------------------------------------------------------------------ helpers */
struct BodyV
{
	float vx, vy, w;
};

struct RowAdj
{
	float n[2];
	float rA[2][2];
	float rB[2][2];
	float base[2];
	float nMass[2];
	float tMass[2];
	float relVel[2];
	float mu;
	float ni[2];
	float ti[2];
	float pad;
};
static_assert( sizeof( RowAdj ) == ADJ_RADJ * 4, "row adjoint layout" );

__device__ __forceinline__ BodyV bv_of( const DevState& s )
{
	BodyV v;
	v.vx = s.v.x;
	v.vy = s.v.y;
	v.w = s.w;
	return v;
}

/* VJP of the impulse application of the 8-lane path (lane_apply / warm_lane):
 * a.v -= mA P, a.w -= iA cross(rA, P), b.v += mB P, b.w += iB cross(rB, P). */
__device__ __forceinline__ b2gVec apply_vjp( b2gVec P, b2gVec rA, b2gVec rB, const Row& r, const BodyV& aA, const BodyV& aB, float* rAbar,
											 float* rBbar )
{
	b2gVec Pb;
	Pb.x = r.mB * aB.vx - r.mA * aA.vx + r.iB * aB.w * ( -rB.y ) - r.iA * aA.w * ( -rA.y );
	Pb.y = r.mB * aB.vy - r.mA * aA.vy + r.iB * aB.w * rB.x - r.iA * aA.w * rA.x;
	rAbar[0] += -r.iA * aA.w * P.y;
	rAbar[1] += r.iA * aA.w * P.x;
	rBbar[0] += r.iB * aB.w * P.y;
	rBbar[1] += -r.iB * aB.w * P.x;
	return Pb;
}

/* VJP of the lane relative velocity dv = (vB + wB x rB) - (vA + wA x rA). */
__device__ __forceinline__ void dv_vjp( b2gVec g, b2gVec rA, b2gVec rB, float wA, float wB, BodyV& aA, BodyV& aB, float* rAbar, float* rBbar )
{
	aB.vx += g.x;
	aB.vy += g.y;
	aA.vx -= g.x;
	aA.vy -= g.y;
	aB.w += -rB.y * g.x + rB.x * g.y;
	aA.w -= -rA.y * g.x + rA.x * g.y;
	rBbar[0] += wB * g.y;
	rBbar[1] += -wB * g.x;
	rAbar[0] -= wA * g.y;
	rAbar[1] -= -wA * g.x;
}

__device__ __forceinline__ b2gVec lane_dv( const DevState& a, const DevState& b, b2gVec aA, b2gVec aB )
{
	float dvx = ( b.v.x - b.w * aB.y ) - ( a.v.x - a.w * aA.y );
	float dvy = ( b.v.y + b.w * aB.x ) - ( a.v.y + a.w * aA.x );
	return gv( dvx, dvy );
}

/* ------------------------------------------------------------------ row VJPs */
/* Warm start (linear in the impulses). */
__device__ void warm_vjp( const Row& r, const BodyV& aA, const BodyV& aB, RowAdj& ra )
{
	b2gVec n = r.n;
	b2gVec t = gv( n.y, 0.0f - n.x );
	for ( int j = 0; j < 2; ++j )
	{
		b2gVec P = gv( r.ni[j] * n.x + r.ti[j] * t.x, r.ni[j] * n.y + r.ti[j] * t.y );
		b2gVec Pb = apply_vjp( P, r.rA[j], r.rB[j], r, aA, aB, ra.rA[j], ra.rB[j] );
		ra.ni[j] += Pb.x * n.x + Pb.y * n.y;
		ra.ti[j] += Pb.x * t.x + Pb.y * t.y;
		ra.n[0] += r.ni[j] * Pb.x - r.ti[j] * Pb.y;
		ra.n[1] += r.ni[j] * Pb.y + r.ti[j] * Pb.x;
	}
}

/* The velocities before each of the row's four impulses (two normal, two friction), from
 * the impulses and velocities before the row.  scalar: an overflow row, whose speculative
 * points (s > 0) take the rigid mass and no impulse scaling where the 8-lane rows keep
 * the soft ones (reference src/contact_solver.c:266-279 against :905-925). */
__device__ __forceinline__ void solve_trace( Row r, DevState a, DevState b, bool useBias, const b2gStepConst& sc, bool scalar, DevState* sa,
											 DevState* sb )
{
	float biasRate = useBias ? r.biasRate : 0.0f;
	float massScale = useBias ? r.massScale : 1.0f;
	float impulseScale = useBias ? r.impulseScale : 0.0f;
	float minBias = -sc.pushout;
	b2gVec n = r.n;
	b2gVec t = gv( n.y, 0.0f - n.x );
	b2gVec dp = gv( b.dp.x - a.dp.x, b.dp.y - a.dp.y );
#pragma unroll
	for ( int j = 0; j < 2; ++j )
	{
		sa[j] = a;
		sb[j] = b;
		b2gVec aA_ = r.rA[j], aB_ = r.rB[j];
		b2gVec rsA = gv( a.dq.c * aA_.x - a.dq.s * aA_.y, a.dq.s * aA_.x + a.dq.c * aA_.y );
		b2gVec rsB = gv( b.dq.c * aB_.x - b.dq.s * aB_.y, b.dq.s * aB_.x + b.dq.c * aB_.y );
		b2gVec ds = gv( dp.x + ( rsB.x - rsA.x ), dp.y + ( rsB.y - rsA.y ) );
		float s = ( n.x * ds.x + n.y * ds.y ) + r.base[j];
		float bias = s > 0.0f ? s * sc.inv_h : gmax( biasRate * s, minBias );
		float ms = scalar && s > 0.0f ? 1.0f : massScale;
		float is = scalar && s > 0.0f ? 0.0f : impulseScale;
		b2gVec dv = lane_dv( a, b, aA_, aB_ );
		float vn = dv.x * n.x + dv.y * n.y;
		float negImpulse = r.nMass[j] * ( ms * ( vn + bias ) ) + is * r.ni[j];
		float newImpulse = gmax( r.ni[j] - negImpulse, 0.0f );
		float impulse = newImpulse - r.ni[j];
		r.ni[j] = newImpulse;
		lane_apply( a, b, r, aA_, aB_, impulse * n.x, impulse * n.y );
	}
#pragma unroll
	for ( int j = 0; j < 2; ++j )
	{
		sa[2 + j] = a;
		sb[2 + j] = b;
		b2gVec aA_ = r.rA[j], aB_ = r.rB[j];
		b2gVec dv = lane_dv( a, b, aA_, aB_ );
		float vt = dv.x * t.x + dv.y * t.y;
		float negImpulse = r.tMass[j] * vt;
		float maxFriction = r.friction * r.ni[j];
		float x = r.ti[j] - negImpulse;
		float lo = 0.0f - maxFriction;
		float mn = x < maxFriction ? x : maxFriction;
		float newImpulse = lo > mn ? lo : mn;
		float impulse = newImpulse - r.ti[j];
		r.ti[j] = newImpulse;
		lane_apply( a, b, r, aA_, aB_, impulse * t.x, impulse * t.y );
	}
}

/* What the reverse of solve / relax needs of that trace and of the row: nothing here
 * depends on an adjoint, so the rows of all colours take it at once. */
struct SolveForward
{
	float impulseN[2], impulseT[2];
	float innerN[2];		/* massScale ( vn + bias ) */
	float massScale[2], impulseScale[2], dbds[2];
	float vt[2], frictionNi[2]; /* friction's relative velocity and normal impulse */
	bool active[2];			/* normal impulse above zero */
	int clampT[2];			/* friction: 0 interior, 1 upper, -1 lower */
	b2gVec dvN[2], dvT[2], ds[2];
	float wA[4], wB[4];
	b2gRot dqA, dqB;
};

/* r holds the impulses before the row ran; sa, sb the states before each impulse, with the
 * substep's position deltas. */
__device__ __forceinline__ void solve_forward( Row r, const DevState* sa, const DevState* sb, bool useBias, const b2gStepConst& sc, bool scalar,
											   SolveForward& F )
{
	float biasRate = useBias ? r.biasRate : 0.0f;
	float massScale = useBias ? r.massScale : 1.0f;
	float impulseScale = useBias ? r.impulseScale : 0.0f;
	float minBias = -sc.pushout;
	b2gVec n = r.n;
	b2gVec t = gv( n.y, 0.0f - n.x );
	b2gVec dp = gv( sb[0].dp.x - sa[0].dp.x, sb[0].dp.y - sa[0].dp.y );
	F.dqA = sa[0].dq;
	F.dqB = sb[0].dq;
#pragma unroll
	for ( int j = 0; j < 2; ++j )
	{
		const DevState& a = sa[j];
		const DevState& b = sb[j];
		b2gVec aA_ = r.rA[j], aB_ = r.rB[j];
		b2gVec rsA = gv( a.dq.c * aA_.x - a.dq.s * aA_.y, a.dq.s * aA_.x + a.dq.c * aA_.y );
		b2gVec rsB = gv( b.dq.c * aB_.x - b.dq.s * aB_.y, b.dq.s * aB_.x + b.dq.c * aB_.y );
		b2gVec ds = gv( dp.x + ( rsB.x - rsA.x ), dp.y + ( rsB.y - rsA.y ) );
		float s = ( n.x * ds.x + n.y * ds.y ) + r.base[j];
		float bias;
		if ( s > 0.0f )
		{
			bias = s * sc.inv_h;
			F.dbds[j] = sc.inv_h;
		}
		else
		{
			float soft = biasRate * s;
			bias = gmax( soft, minBias );
			F.dbds[j] = soft > minBias ? biasRate : 0.0f;
		}
		F.ds[j] = ds;
		F.massScale[j] = scalar && s > 0.0f ? 1.0f : massScale;
		F.impulseScale[j] = scalar && s > 0.0f ? 0.0f : impulseScale;
		b2gVec dv = lane_dv( a, b, aA_, aB_ );
		F.dvN[j] = dv;
		float vn = dv.x * n.x + dv.y * n.y;
		F.innerN[j] = F.massScale[j] * ( vn + bias );
		float negImpulse = r.nMass[j] * F.innerN[j] + F.impulseScale[j] * r.ni[j];
		float x = r.ni[j] - negImpulse;
		float newImpulse = gmax( x, 0.0f );
		F.active[j] = x > 0.0f;
		F.impulseN[j] = newImpulse - r.ni[j];
		F.frictionNi[j] = newImpulse;
		F.wA[j] = a.w;
		F.wB[j] = b.w;
	}
#pragma unroll
	for ( int j = 0; j < 2; ++j )
	{
		b2gVec dv = lane_dv( sa[2 + j], sb[2 + j], r.rA[j], r.rB[j] );
		float vt = dv.x * t.x + dv.y * t.y;
		float negImpulse = r.tMass[j] * vt;
		float maxFriction = r.friction * F.frictionNi[j];
		float x = r.ti[j] - negImpulse;
		float lo = 0.0f - maxFriction;
		float mn = x < maxFriction ? x : maxFriction;
		F.clampT[j] = lo > mn ? -1 : ( x < maxFriction ? 0 : 1 );
		float newImpulse = F.clampT[j] < 0 ? -maxFriction : ( F.clampT[j] == 0 ? x : maxFriction );
		F.impulseT[j] = newImpulse - r.ti[j];
		F.dvT[j] = dv;
		F.vt[j] = vt;
		F.wA[2 + j] = sa[2 + j].w;
		F.wB[2 + j] = sb[2 + j].w;
	}
}

/* Reverse of solve / relax.  On entry aA, aB are the adjoints of the velocities after the
 * row; on exit, before it.  dpA.. receive the position-delta adjoints. */
__device__ __forceinline__ void solve_reverse( const Row& r, const SolveForward& F, BodyV& aA, BodyV& aB, RowAdj& ra, float* dpA, float* dqA,
											   float* dpB, float* dqB )
{
	b2gVec n = r.n;
	b2gVec t = gv( n.y, 0.0f - n.x );
	/* tangent points in reverse */
#pragma unroll
	for ( int j = 1; j >= 0; --j )
	{
		float impulse = F.impulseT[j];
		b2gVec P = gv( impulse * t.x, impulse * t.y );
		b2gVec Pb = apply_vjp( P, r.rA[j], r.rB[j], r, aA, aB, ra.rA[j], ra.rB[j] );
		float impb = Pb.x * t.x + Pb.y * t.y;
		ra.n[0] += -( impulse * Pb.y );
		ra.n[1] += impulse * Pb.x;
		float newb = ra.ti[j] + impb;
		float tib = -impb;
		float xb = 0.0f, maxFb = 0.0f;
		if ( F.clampT[j] < 0 )
			maxFb = -newb;
		else if ( F.clampT[j] == 0 )
			xb = newb;
		else
			maxFb = newb;
		ra.mu += maxFb * F.frictionNi[j];
		ra.ni[j] += maxFb * r.friction;
		tib += xb;
		float negb = -xb;
		b2gVec dv = F.dvT[j];
		ra.tMass[j] += negb * F.vt[j];
		float vtb = negb * r.tMass[j];
		/* vt = dv . t, t = ( n.y, -n.x ) */
		ra.n[0] += -( vtb * dv.y );
		ra.n[1] += vtb * dv.x;
		dv_vjp( gv( vtb * t.x, vtb * t.y ), r.rA[j], r.rB[j], F.wA[2 + j], F.wB[2 + j], aA, aB, ra.rA[j], ra.rB[j] );
		ra.ti[j] = tib;
	}
	/* normal points in reverse */
#pragma unroll
	for ( int j = 1; j >= 0; --j )
	{
		float impulse = F.impulseN[j];
		b2gVec P = gv( impulse * n.x, impulse * n.y );
		b2gVec Pb = apply_vjp( P, r.rA[j], r.rB[j], r, aA, aB, ra.rA[j], ra.rB[j] );
		float impb = Pb.x * n.x + Pb.y * n.y;
		ra.n[0] += impulse * Pb.x;
		ra.n[1] += impulse * Pb.y;
		float newb = ra.ni[j] + impb;
		float nib = -impb;
		float xb = F.active[j] ? newb : 0.0f;
		nib += xb;
		float negb = -xb;
		b2gVec dv = F.dvN[j];
		/* negImpulse = nMass * ( massScale * ( vn + bias ) ) + impulseScale * ni */
		ra.nMass[j] += negb * F.innerN[j];
		float vnb = negb * r.nMass[j] * F.massScale[j];
		nib += negb * F.impulseScale[j];
		float sb_ = vnb * F.dbds[j];
		ra.n[0] += vnb * dv.x;
		ra.n[1] += vnb * dv.y;
		dv_vjp( gv( vnb * n.x, vnb * n.y ), r.rA[j], r.rB[j], F.wA[j], F.wB[j], aA, aB, ra.rA[j], ra.rB[j] );
		/* s = n . ( dp + rotate( dqB, rB ) - rotate( dqA, rA ) ) + base */
		b2gVec aA_ = r.rA[j], aB_ = r.rB[j];
		ra.n[0] += sb_ * F.ds[j].x;
		ra.n[1] += sb_ * F.ds[j].y;
		ra.base[j] += sb_;
		b2gVec dsb = gv( sb_ * n.x, sb_ * n.y );
		dpB[0] += dsb.x;
		dpB[1] += dsb.y;
		dpA[0] -= dsb.x;
		dpA[1] -= dsb.y;
		/* rotate( q, v ): d/dq.c = v, d/dq.s = ( -v.y, v.x ); d/dv = rotate^T */
		dqB[0] += dsb.x * aB_.x + dsb.y * aB_.y;
		dqB[1] += -dsb.x * aB_.y + dsb.y * aB_.x;
		dqA[0] -= dsb.x * aA_.x + dsb.y * aA_.y;
		dqA[1] -= -dsb.x * aA_.y + dsb.y * aA_.x;
		ra.rB[j][0] += F.dqB.c * dsb.x + F.dqB.s * dsb.y;
		ra.rB[j][1] += -F.dqB.s * dsb.x + F.dqB.c * dsb.y;
		ra.rA[j][0] -= F.dqA.c * dsb.x + F.dqA.s * dsb.y;
		ra.rA[j][1] -= -F.dqA.s * dsb.x + F.dqA.c * dsb.y;
		ra.ni[j] = nib;
	}
}

/* Solve / relax from the states before the row: trace, then reverse. */
__device__ void solve_vjp( Row r, DevState a, DevState b, bool useBias, const b2gStepConst& sc, BodyV& aA, BodyV& aB, RowAdj& ra,
						   float* dpA, float* dqA, float* dpB, float* dqB, bool scalar = false )
{
	DevState sa[4], sb[4];
	solve_trace( r, a, b, useBias, sc, scalar, sa, sb );
	SolveForward F;
	solve_forward( r, sa, sb, useBias, sc, scalar, F );
	solve_reverse( r, F, aA, aB, ra, dpA, dqA, dpB, dqB );
}

/* Restitution (8-lane path): the states before its two impulses, and its reverse. */
__device__ __forceinline__ void restitution_trace( Row r, DevState a, DevState b, const b2gStepConst& sc, DevState* sa, DevState* sb )
{
	b2gVec n = r.n;
#pragma unroll
	for ( int j = 0; j < 2; ++j )
	{
		sa[j] = a;
		sb[j] = b;
		bool skip = ( r.relVel[j] + sc.restitutionThreshold > 0.0f ) || ( r.maxNi[j] == 0.0f );
		float mass = skip ? 0.0f : r.nMass[j];
		b2gVec dv = lane_dv( a, b, r.rA[j], r.rB[j] );
		float vn = dv.x * n.x + dv.y * n.y;
		float negImpulse = mass * ( vn + r.restitution * r.relVel[j] );
		float newImpulse = gmax( r.ni[j] - negImpulse, 0.0f );
		float impulse = newImpulse - r.ni[j];
		lane_apply( a, b, r, r.rA[j], r.rB[j], impulse * n.x, impulse * n.y );
	}
}

__device__ __forceinline__ void restitution_reverse( Row r, const DevState* sa, const DevState* sb, const b2gStepConst& sc, BodyV& aA, BodyV& aB,
													 RowAdj& ra )
{
	b2gVec n = r.n;
	float xN[2], ni0[2] = { r.ni[0], r.ni[1] }, mass[2];
#pragma unroll
	for ( int j = 0; j < 2; ++j )
	{
		bool skip = ( r.relVel[j] + sc.restitutionThreshold > 0.0f ) || ( r.maxNi[j] == 0.0f );
		mass[j] = skip ? 0.0f : r.nMass[j];
		b2gVec dv = lane_dv( sa[j], sb[j], r.rA[j], r.rB[j] );
		float vn = dv.x * n.x + dv.y * n.y;
		float negImpulse = mass[j] * ( vn + r.restitution * r.relVel[j] );
		xN[j] = r.ni[j] - negImpulse;
	}
#pragma unroll
	for ( int j = 1; j >= 0; --j )
	{
		const DevState& A = sa[j];
		const DevState& B = sb[j];
		float newImpulse = gmax( xN[j], 0.0f );
		float impulse = newImpulse - ni0[j];
		b2gVec P = gv( impulse * n.x, impulse * n.y );
		b2gVec Pb = apply_vjp( P, r.rA[j], r.rB[j], r, aA, aB, ra.rA[j], ra.rB[j] );
		float impb = Pb.x * n.x + Pb.y * n.y;
		ra.n[0] += impulse * Pb.x;
		ra.n[1] += impulse * Pb.y;
		float newb = ra.ni[j] + impb;
		float nib = -impb;
		float xb = xN[j] > 0.0f ? newb : 0.0f;
		nib += xb;
		float negb = -xb;
		b2gVec dv = lane_dv( A, B, r.rA[j], r.rB[j] );
		float vn = dv.x * n.x + dv.y * n.y;
		if ( mass[j] != 0.0f )
			ra.nMass[j] += negb * ( vn + r.restitution * r.relVel[j] );
		float inner = negb * mass[j];
		ra.relVel[j] += inner * r.restitution;
		ra.n[0] += inner * dv.x;
		ra.n[1] += inner * dv.y;
		dv_vjp( gv( inner * n.x, inner * n.y ), r.rA[j], r.rB[j], A.w, B.w, aA, aB, ra.rA[j], ra.rB[j] );
		ra.ni[j] = nib;
	}
}

__device__ void restitution_vjp( Row r, DevState a, DevState b, const b2gStepConst& sc, BodyV& aA, BodyV& aB, RowAdj& ra )
{
	DevState sa[2], sb[2];
	restitution_trace( r, a, b, sc, sa, sb );
	restitution_reverse( r, sa, sb, sc, aA, aB, ra );
}

/* ------------------------------------------------------------------ body VJPs */
/* Body adjoint layout (12 floats): c.x c.y q.c q.s | v.x v.y w | dp.x dp.y | dq.c dq.s | - */

/* integrate_velocity: v' = cap( lvd + ld v ), w' = cap( avd + ad w ) */
__device__ void iv_vjp( const float* pre, float4 term, float ad, const b2gStepConst& sc, float* g )
{
	float maxLin = B2G_MAX_TRANSLATION * sc.inv_dt;
	float maxAng = B2G_MAX_ROTATION * sc.inv_dt;
	b2gVec v = gmuladd( gv( term.x, term.y ), term.w, gv( pre[0], pre[1] ) );
	float w = term.z + ad * pre[2];
	float gx = g[4], gy = g[5], gw = g[6];
	if ( gdot( v, v ) > maxLin * maxLin )
	{
		float L = glen( v );
		float k = maxLin / L;
		b2gVec u = gv( v.x / L, v.y / L );
		float d = gx * u.x + gy * u.y;
		gx = k * ( gx - d * u.x );
		gy = k * ( gy - d * u.y );
	}
	if ( w * w > maxAng * maxAng )
		gw = 0.0f;
	g[4] = term.w * gx;
	g[5] = term.w * gy;
	g[6] = ad * gw;
}

/* integrate_position: dq' = normalize( dq + h w perp( dq ) ), dp' = dp + h v */
__device__ void ip_vjp( const float* pre, float h, float* g )
{
	float dqc = pre[6], dqs = pre[7];
	float da = h * pre[2];
	float q2c = dqc - da * dqs, q2s = dqs + da * dqc;
	float mag = sqrtf( q2s * q2s + q2c * q2c );
	float inv = mag > 0.0f ? 1.0f / mag : 0.0f;
	float nc = q2c * inv, ns = q2s * inv;
	float d = nc * g[9] + ns * g[10];
	float g2c = ( g[9] - nc * d ) * inv, g2s = ( g[10] - ns * d ) * inv;
	g[9] = g2c + da * g2s;
	g[10] = -da * g2c + g2s;
	g[6] += h * ( -dqs * g2c + dqc * g2s );
	g[4] += h * g[7];
	g[5] += h * g[8];
}

/* finalisation: c' = c + dp, q' = normalize( dq q ) (reference src/solver.c:205-223) */
__device__ void finalize_vjp( float qc, float qs, float dqc, float dqs, float* g )
{
	float us = dqs * qc + dqc * qs;
	float uc = dqc * qc - dqs * qs;
	float mag = sqrtf( us * us + uc * uc );
	float inv = mag > 0.0f ? 1.0f / mag : 0.0f;
	float nc = uc * inv, ns = us * inv;
	float d = nc * g[2] + ns * g[3];
	float guc = ( g[2] - nc * d ) * inv, gus = ( g[3] - ns * d ) * inv;
	g[9] = guc * qc + gus * qs;
	g[10] = -guc * qs + gus * qc;
	g[2] = guc * dqc + gus * dqs;
	g[3] = -guc * dqs + gus * dqc;
	g[7] = g[0];
	g[8] = g[1];
}

/* ------------------------------------------------------------------ prepare VJP */
/* Adjoint of the row preparation (reference src/contact_solver.c:597-808) with
 * respect to the manifold (normal, centre-relative anchors, separations), the bodies'
 * step-start velocities and the warm-start impulses.  mAdj: n(2), then per point
 * anchorA(2) anchorB(2) separation. */
/* The part that does not add to the bodies' velocity adjoints, whose terms of point j are
 * those of dv_vjp for g[j]. */
__device__ __forceinline__ void prepare_parts( const Row& r, const DevState& sA, const DevState& sB, const RowAdj& ra, float warm, float* mAdj,
											   b2gVec* g, float* lamIn )
{
	b2gVec n = r.n;
	b2gVec t = gright( n );
	float nb[2] = { ra.n[0], ra.n[1] };
	float tb[2] = { 0.0f, 0.0f };
	for ( int i = 0; i < 12; ++i )
		mAdj[i] = 0.0f;
	for ( int i = 0; i < 4; ++i )
		lamIn[i] = 0.0f;
#pragma unroll
	for ( int j = 0; j < 2; ++j )
	{
		g[j] = gv( 0.0f, 0.0f );
		if ( j >= r.count )
			continue;
		b2gVec rA = r.rA[j], rB = r.rB[j];
		float rAb[2] = { ra.rA[j][0], ra.rA[j][1] };
		float rBb[2] = { ra.rB[j][0], ra.rB[j][1] };
		/* base = separation - ( rB - rA ) . n */
		float gb = ra.base[j];
		float sepb = gb;
		rBb[0] -= gb * n.x;
		rBb[1] -= gb * n.y;
		rAb[0] += gb * n.x;
		rAb[1] += gb * n.y;
		nb[0] -= gb * ( rB.x - rA.x );
		nb[1] -= gb * ( rB.y - rA.y );
		/* normal and tangent mass: 1 / ( mA + mB + iA rn_A^2 + iB rn_B^2 ) */
		if ( r.nMass[j] > 0.0f )
		{
			float rnA = gcross( rA, n ), rnB = gcross( rB, n );
			float gk = -ra.nMass[j] * r.nMass[j] * r.nMass[j];
			float grA = gk * 2.0f * r.iA * rnA, grB = gk * 2.0f * r.iB * rnB;
			rAb[0] += grA * n.y;
			rAb[1] += -grA * n.x;
			nb[0] += -grA * rA.y;
			nb[1] += grA * rA.x;
			rBb[0] += grB * n.y;
			rBb[1] += -grB * n.x;
			nb[0] += -grB * rB.y;
			nb[1] += grB * rB.x;
		}
		if ( r.tMass[j] > 0.0f )
		{
			float rtA = gcross( rA, t ), rtB = gcross( rB, t );
			float gk = -ra.tMass[j] * r.tMass[j] * r.tMass[j];
			float grA = gk * 2.0f * r.iA * rtA, grB = gk * 2.0f * r.iB * rtB;
			rAb[0] += grA * t.y;
			rAb[1] += -grA * t.x;
			tb[0] += -grA * rA.y;
			tb[1] += grA * rA.x;
			rBb[0] += grB * t.y;
			rBb[1] += -grB * t.x;
			tb[0] += -grB * rB.y;
			tb[1] += grB * rB.x;
		}
		/* relative normal velocity at the step start */
		float gr = ra.relVel[j];
		b2gVec dv = gsub( gadd( sB.v, gcross_sv( sB.w, rB ) ), gadd( sA.v, gcross_sv( sA.w, rA ) ) );
		nb[0] += gr * dv.x;
		nb[1] += gr * dv.y;
		g[j] = gv( gr * n.x, gr * n.y );
		rBb[0] += sB.w * g[j].y;
		rBb[1] += -sB.w * g[j].x;
		rAb[0] -= sA.w * g[j].y;
		rAb[1] -= -sA.w * g[j].x;
		lamIn[j] = warm * ra.ni[j];
		lamIn[2 + j] = warm * ra.ti[j];
		mAdj[2 + 5 * j + 0] = rAb[0];
		mAdj[2 + 5 * j + 1] = rAb[1];
		mAdj[2 + 5 * j + 2] = rBb[0];
		mAdj[2 + 5 * j + 3] = rBb[1];
		mAdj[2 + 5 * j + 4] = sepb;
	}
	/* t = ( n.y, -n.x ) */
	nb[0] += -tb[1];
	nb[1] += tb[0];
	mAdj[0] = nb[0];
	mAdj[1] = nb[1];
}

/* The velocity terms of dv_vjp for g. */
__device__ __forceinline__ void dv_velocities( b2gVec g, b2gVec rA, b2gVec rB, BodyV& aA, BodyV& aB )
{
	aB.vx += g.x;
	aB.vy += g.y;
	aA.vx -= g.x;
	aA.vy -= g.y;
	aB.w += -rB.y * g.x + rB.x * g.y;
	aA.w -= -rA.y * g.x + rA.x * g.y;
}

__device__ void prepare_vjp( const Row& r, const DevState& sA, const DevState& sB, const RowAdj& ra, float warm, float* mAdj, BodyV& aA,
							 BodyV& aB, float* lamIn )
{
	b2gVec g[2];
	prepare_parts( r, sA, sB, ra, warm, mAdj, g, lamIn );
	for ( int j = 0; j < r.count; ++j )
		dv_velocities( g[j], r.rA[j], r.rB[j], aA, aB );
}

/* ------------------------------------------------------------------ narrowphase Jacobian */
/* Recomputes the manifold of a polygon pair with derivatives in the six directions
 * ( cA.x, cA.y, angleA, cB.x, cB.y, angleB ); writes the 12 x 6 Jacobian of
 * ( normal, per point anchorA anchorB separation ), anchors relative to the centres.
 * Returns false when the replay does not reproduce the recorded manifold. */
__device__ bool manifold_jacobian( const b2gShapeGeo& gA, const b2gShapeGeo& gB, const float* startA, const float* startB, bool dynA, bool dynB,
								   const b2gManifold& rec, float* jac, int stride = 1 )
{
	typedef Dual<6> D;
	DXf<6> xf[2];
	const float* st[2] = { startA, startB };
	bool dyn[2] = { dynA, dynB };
	DRot<6> q[2];
	for ( int k = 0; k < 2; ++k )
	{
		/* start record: c.x c.y q.c q.s lc.x lc.y p.x p.y */
		float qc = st[k][2], qs = st[k][3], lcx = st[k][4], lcy = st[k][5];
		D px = dc<6>( st[k][6] ), py = dc<6>( st[k][7] );
		D c = dc<6>( qc ), s = dc<6>( qs );
		if ( dyn[k] )
		{
			int o = 3 * k;
			px.d[o + 0] = 1.0f;
			py.d[o + 1] = 1.0f;
			/* p = c - rotate( q, lc ) */
			px.d[o + 2] = qs * lcx + qc * lcy;
			py.d[o + 2] = -qc * lcx + qs * lcy;
			c.d[o + 2] = -qs;
			s.d[o + 2] = qc;
		}
		xf[k].p = dv( px, py );
		xf[k].q.c = c;
		xf[k].q.s = s;
		q[k] = xf[k].q;
	}
	/* the narrowphase's dispatch (b2g_collide.h gcollide_shapes) for A not a chain link */
	DManifold<6> m;
	if ( gB.type == 0 )
	{
		if ( gA.type == 0 )
			dcollide_circles( m, gA.v[0], gA.radius, xf[0], gB.v[0], gB.radius, xf[1] );
		else if ( gA.type == 1 || gA.type == 2 )
			dcollide_capsule_circle( m, gA.v[0], gA.v[1], gA.type == 1 ? gA.radius : 0.0f, xf[0], gB.v[0], gB.radius, xf[1] );
		else
		{
			b2gPoly pa;
			gshape_poly( &pa, &gA );
			dcollide_polygon_circle( m, pa, xf[0], gB.v[0], gB.radius, xf[1] );
		}
	}
	else
	{
		b2gPoly pa, pb;
		gshape_poly( &pa, &gA );
		gshape_poly( &pb, &gB );
		dcollide_polygons( m, pa, xf[0], pb, xf[1] );
	}
	DVec<6> offA = drotate( q[0], dvc<6>( gv( startA[4], startA[5] ) ) );
	DVec<6> offB = drotate( q[1], dvc<6>( gv( startB[4], startB[5] ) ) );
	bool same = m.count == rec.count && m.normal.x.v == rec.normal.x && m.normal.y.v == rec.normal.y;
	for ( int i = 0; i < 12 * 6; ++i )
		jac[(size_t)i * stride] = 0.0f;
	for ( int d = 0; d < 6; ++d )
	{
		jac[(size_t)( 0 * 6 + d ) * stride] = m.normal.x.d[d];
		jac[(size_t)( 1 * 6 + d ) * stride] = m.normal.y.d[d];
	}
	for ( int j = 0; j < m.count && j < 2; ++j )
	{
		DVec<6> aA = dsub( m.pts[j].anchorA, offA );
		DVec<6> aB = dsub( m.pts[j].anchorB, offB );
		same = same && aA.x.v == rec.pts[j].anchorA.x && aA.y.v == rec.pts[j].anchorA.y && aB.x.v == rec.pts[j].anchorB.x &&
			   aB.y.v == rec.pts[j].anchorB.y && m.pts[j].separation.v == rec.pts[j].separation && m.pts[j].id == rec.pts[j].id;
		for ( int d = 0; d < 6; ++d )
		{
			jac[(size_t)( ( 2 + 5 * j + 0 ) * 6 + d ) * stride] = aA.x.d[d];
			jac[(size_t)( ( 2 + 5 * j + 1 ) * 6 + d ) * stride] = aA.y.d[d];
			jac[(size_t)( ( 2 + 5 * j + 2 ) * 6 + d ) * stride] = aB.x.d[d];
			jac[(size_t)( ( 2 + 5 * j + 3 ) * 6 + d ) * stride] = aB.y.d[d];
			jac[(size_t)( ( 2 + 5 * j + 4 ) * 6 + d ) * stride] = m.pts[j].separation.d[d];
		}
	}
	return same;
}

/* ------------------------------------------------------------------ replay */
#define ADJ_WARP 32
#define ADJ_LINK_NONE 3

__device__ __forceinline__ DevState replay_state( const float* state, int b )
{
	if ( b < 0 )
		return identity_state();
	const float4* s = (const float4*)( state + (size_t)b * ADJ_STATE );
	return state_of( s[0], s[1] );
}

__device__ __forceinline__ void replay_store_velocity( float* state, int b, const DevState& x )
{
	if ( b < 0 )
		return;
	float* s = state + (size_t)b * ADJ_STATE;
	s[0] = x.v.x;
	s[1] = x.v.y;
	s[2] = x.w;
}

__device__ __forceinline__ void put_velocity( float* p, int Rs, const DevState& A, const DevState& B )
{
	p[0] = A.v.x;
	p[Rs] = A.v.y;
	p[2 * Rs] = A.w;
	p[3 * Rs] = B.v.x;
	p[4 * Rs] = B.v.y;
	p[5 * Rs] = B.w;
}

/* One phase of a replayed row (warm 0, solve 1, relax 2, restitution 3): what its reverse
 * starts from onto the phase tape, then the row itself. */
__device__ __forceinline__ void replay_row( const AdjStep& L, float* D, int k, int phase, int sub, const b2gStepConst& sc, bool scalar )
{
	const int Rs = L.Rs;
	float* state = D + L.state;
	Row* work = (Row*)( D + L.work );
	Row r = work[k];
	DevState A = replay_state( state, r.ia );
	DevState B = replay_state( state, r.ib );
	bool changed = true;
	if ( phase == 0 )
	{
		float* t = D + L.warm( sub ) + k;
		t[0] = r.ni[0];
		t[Rs] = r.ni[1];
		t[2 * Rs] = r.ti[0];
		t[3 * Rs] = r.ti[1];
		scalar ? warm_scalar( r, A, B ) : warm_lane( r, A, B );
	}
	else if ( phase == 3 )
	{
		DevState sa[2], sb[2];
		restitution_trace( r, A, B, sc, sa, sb );
		float* t = D + L.rest() + k;
		t[0] = r.ni[0];
		t[Rs] = r.ni[1];
		t[2 * Rs] = r.maxNi[0];
		t[3 * Rs] = r.maxNi[1];
		for ( int j = 0; j < 2; ++j )
			put_velocity( t + ( 4 + 6 * j ) * Rs, Rs, sa[j], sb[j] );
		if ( scalar )
			changed = restitution_scalar( r, A, B, sc.restitutionThreshold );
		else
			restitution_lane( r, A, B, sc.restitutionThreshold );
	}
	else
	{
		DevState sa[4], sb[4];
		solve_trace( r, A, B, phase == 1, sc, scalar, sa, sb );
		float* t = D + L.solve( sub, phase == 2 ) + k;
		t[0] = r.ni[0];
		t[Rs] = r.ni[1];
		t[2 * Rs] = r.ti[0];
		t[3 * Rs] = r.ti[1];
#pragma unroll
		for ( int j = 0; j < 4; ++j )
			put_velocity( t + ( 4 + 6 * j ) * Rs, Rs, sa[j], sb[j] );
		scalar ? solve_scalar( r, A, B, phase == 1, sc.inv_h, sc.pushout ) : solve_lane( r, A, B, phase == 1, sc.inv_h, sc.pushout );
	}
	if ( changed == false )
		return;
	replay_store_velocity( state, r.ia, A );
	replay_store_velocity( state, r.ib, B );
	for ( int j = 0; j < 2; ++j )
	{
		work[k].ni[j] = r.ni[j];
		work[k].ti[j] = r.ti[j];
		work[k].maxNi[j] = r.maxNi[j];
	}
}

/* One forward stage of the replay over the active colours: the overflow colour first, one
 * row after another with the scalar arithmetic (reference src/contact_solver.c:149-440). */
__device__ void replay_stage( const AdjStep& L, float* D, const b2gTapeStep& h, int phase, int sub, const b2gStepConst& sc )
{
	if ( threadIdx.x == 0 )
		for ( int k = h.colorStart[B2G_OVERFLOW]; k < h.colorStart[B2G_COLORS]; ++k )
			replay_row( L, D, k, phase, sub, sc, true );
	__syncwarp();
	for ( int a = 0; a < h.activeCount; ++a )
	{
		int c = h.active[a];
		for ( int k = h.colorStart[c] + (int)threadIdx.x; k < h.colorStart[c + 1]; k += ADJ_WARP )
			replay_row( L, D, k, phase, sub, sc, false );
		__syncwarp();
	}
}

__device__ void snapshot( const AdjStep& L, float* D, int N, int index )
{
	float* dst = D + L.snap + (size_t)index * ADJ_SNAP * L.Ns;
	for ( int b = threadIdx.x; b < N; b += ADJ_WARP )
		for ( int i = 0; i < ADJ_SNAP; ++i )
			dst[(size_t)i * L.Ns + b] = D[L.state + (size_t)b * ADJ_STATE + i];
	__syncwarp();
}

/* Block n i + t of a chunk of n steps: the replay of step stepCount - 1 - (first + t) of
 * world i.  Reads the tape and the world; writes that step's scratch and, added, the
 * world's status. */
__global__ void __launch_bounds__( ADJ_WARP ) k_adjoint_replay( const b2gAdjointItem* items, int first, int n )
{
	const int t = (int)( blockIdx.x % (unsigned)n );
	const b2gAdjointItem& it = items[blockIdx.x / (unsigned)n];
	const int ts = it.stepCount - 1 - ( first + t );
	if ( ts < 0 )
		return;
	const b2gDevWorld& W = it.W;
	const int lane = threadIdx.x;
	const int N = it.bodies;
	const AdjStep L = adj_step( N, it.maxRows, it.maxSub );
	float* D = it.stepScratch + (size_t)t * it.stepFloats;
	int* table = (int*)( D + L.total ); /* rows of the step before by contact id, where set */
	const b2gTapeStep& h = it.steps[ts];
	const b2gStepConst& sc = h.sc;
	const int R = h.rows, Rs = L.Rs, Ns = L.Ns;
	const int S = sc.subSteps;
	int unsupported = 0, mismatches = 0, replayDiffs = 0;
	if ( h.solve == 0 || S > ADJ_MAX_SUBSTEPS )
	{
		if ( h.solve != 0 && lane == 0 )
			atomicAdd( it.status, 1 );
		return;
	}
	if ( h.jointStart[B2G_COLORS] > 0 )
		unsupported += 1;
	const float* recB = it.tapeBodies + 4 * h.bodyOff;
	const b2gTapeRow* recR = it.tapeRows + h.rowOff;
	const b2gTapeRow* oldR = it.tapeRows;
	int oldRows = 0;
	if ( ts > 0 )
	{
		oldR = it.tapeRows + it.steps[ts - 1].rowOff;
		oldRows = it.steps[ts - 1].rows;
		for ( int k = lane; k < oldRows; k += ADJ_WARP )
			table[oldR[k].cid] = k;
	}

	/* step start: bodies */
	for ( int b = lane; b < N; b += ADJ_WARP )
	{
		const float* o = recB + 16 * b;
		float* st = D + L.start + b;
		st[0 * Ns] = o[8];
		st[1 * Ns] = o[9];
		st[2 * Ns] = o[6];
		st[3 * Ns] = o[7];
		st[4 * Ns] = o[10];
		st[5 * Ns] = o[11];
		st[6 * Ns] = o[4];
		st[7 * Ns] = o[5];
		st[8 * Ns] = o[12];
		float4* x = (float4*)( D + L.state + (size_t)b * ADJ_STATE );
		x[0] = make_float4( o[0], o[1], o[2], o[3] );
		x[1] = make_float4( 0.0f, 0.0f, 1.0f, 0.0f );
		if ( o[12] != 0.0f )
		{
			float4 ms = ( (const float4*)W.mass )[b];
			float4 fo = ( (const float4*)W.force )[b];
			fo = make_float4( o[13], o[14], o[15], fo.w );
			float4 ex = ( (const float4*)W.extent )[b];
			VelocityTerms v = velocity_terms( ms, fo, ex, sc );
			float* tm = D + L.terms + b;
			tm[0 * Ns] = v.lvd.x;
			tm[1 * Ns] = v.lvd.y;
			tm[2 * Ns] = v.avd;
			tm[3 * Ns] = v.ld;
			tm[4 * Ns] = v.ad;
		}
	}
	__syncwarp();

	/* rows: manifold Jacobian, preparation, the previous step's row and points */
	const float4* mass = (const float4*)W.mass;
	for ( int k = lane; k < R; k += ADJ_WARP )
	{
		const b2gTapeRow& tr = recR[k];
		const b2gShapeGeo& gA = W.geo[tr.shapeA];
		const b2gShapeGeo& gB = W.geo[tr.shapeB];
		float startA[8], startB[8];
		for ( int i = 0; i < 8; ++i )
		{
			startA[i] = D[L.start + (size_t)i * Ns + gA.bodyId];
			startB[i] = D[L.start + (size_t)i * Ns + gB.bodyId];
		}
		if ( gA.type == 4 )
			unsupported += 1; /* chain links have no manifold Jacobian here */
		else if ( manifold_jacobian( gA, gB, startA, startB, tr.ia >= 0, tr.ib >= 0, tr.m, D + L.jac + k, Rs ) == false )
			mismatches += 1;
		float4 zero = make_float4( 0.0f, 0.0f, 0.0f, 0.0f );
		Row r;
		prepare_row( r, &tr.m, tr.ia, tr.ib, tr.ia >= 0 ? mass[tr.ia] : zero, tr.ib >= 0 ? mass[tr.ib] : zero,
					 replay_state( D + L.state, tr.ia ), replay_state( D + L.state, tr.ib ), tr.friction, tr.restitution,
					 ( tr.ia < 0 || tr.ib < 0 ) ? sc.staticSoft : sc.contactSoft, sc.enableWarmStarting ? 1.0f : 0.0f );
		( (Row*)( D + L.work ) )[k] = r;
		/* warm-start impulses came from the previous step's stored impulses of the points
		 * with the same feature id (reference src/contact.c:555-568) */
		int link = -1;
		if ( oldRows > 0 )
		{
			int o = table[tr.cid];
			if ( o >= 0 && o < oldRows && oldR[o].cid == tr.cid )
			{
				const b2gTapeRow& old = oldR[o];
				int from[2] = { ADJ_LINK_NONE, ADJ_LINK_NONE };
				for ( int j = 0; j < tr.m.count; ++j )
					for ( int jo = old.m.count - 1; jo >= 0; --jo )
						if ( old.m.pts[jo].id == tr.m.pts[j].id )
							from[j] = jo;
				link = o | ( from[0] << 24 ) | ( from[1] << 26 );
			}
		}
		float* f = D + L.rows + k;
		f[0 * Rs] = __int_as_float( r.ia );
		f[1 * Rs] = __int_as_float( r.ib );
		f[2 * Rs] = __int_as_float( r.count );
		f[3 * Rs] = r.n.x;
		f[4 * Rs] = r.n.y;
		f[5 * Rs] = r.friction;
		f[6 * Rs] = r.restitution;
		f[7 * Rs] = r.mA;
		f[8 * Rs] = r.iA;
		f[9 * Rs] = r.mB;
		f[10 * Rs] = r.iB;
		for ( int j = 0; j < 2; ++j )
		{
			f[( 11 + 2 * j ) * Rs] = r.rA[j].x;
			f[( 12 + 2 * j ) * Rs] = r.rA[j].y;
			f[( 15 + 2 * j ) * Rs] = r.rB[j].x;
			f[( 16 + 2 * j ) * Rs] = r.rB[j].y;
			f[( 19 + j ) * Rs] = r.base[j];
			f[( 21 + j ) * Rs] = r.nMass[j];
			f[( 23 + j ) * Rs] = r.tMass[j];
			f[( 25 + j ) * Rs] = r.relVel[j];
		}
		f[27 * Rs] = __int_as_float( link );
	}
	__syncwarp();

	for ( int sub = 0; sub < S; ++sub )
	{
		snapshot( L, D, N, 2 * sub );
		for ( int b = lane; b < N; b += ADJ_WARP )
		{
			if ( D[L.start + 8 * Ns + b] == 0.0f )
				continue;
			DevState x = replay_state( D + L.state, b );
			const float* tm = D + L.terms + b;
			VelocityTerms v;
			v.lvd = gv( tm[0 * Ns], tm[1 * Ns] );
			v.avd = tm[2 * Ns];
			v.ld = tm[3 * Ns];
			v.ad = tm[4 * Ns];
			integrate_velocity( x, v, sc );
			replay_store_velocity( D + L.state, b, x );
		}
		__syncwarp();
		if ( sc.enableWarmStarting )
			replay_stage( L, D, h, 0, sub, sc );
		replay_stage( L, D, h, 1, sub, sc );
		snapshot( L, D, N, 2 * sub + 1 );
		for ( int b = lane; b < N; b += ADJ_WARP )
		{
			if ( D[L.start + 8 * Ns + b] == 0.0f )
				continue;
			DevState x = replay_state( D + L.state, b );
			integrate_position( x, sc.h );
			( (float4*)( D + L.state + (size_t)b * ADJ_STATE ) )[1] = make_float4( x.dp.x, x.dp.y, x.dq.c, x.dq.s );
		}
		__syncwarp();
		replay_stage( L, D, h, 2, sub, sc );
	}
	snapshot( L, D, N, 2 * S );
	replay_stage( L, D, h, 3, 0, sc );

	/* the replayed step must end where the next recorded step starts */
	if ( ts + 1 < it.stepCount )
	{
		const float* next = it.tapeBodies + 4 * it.steps[ts + 1].bodyOff;
		for ( int b = lane; b < N; b += ADJ_WARP )
		{
			const float* st = D + L.start + b;
			if ( st[8 * Ns] == 0.0f )
				continue;
			const float* x = D + L.state + (size_t)b * ADJ_STATE;
			const float* o = next + 16 * b;
			b2gRot qf = gnormrot( gmulrot( grot( x[6], x[7] ), grot( st[2 * Ns], st[3 * Ns] ) ) );
			bool same = x[0] == o[0] && x[1] == o[1] && x[2] == o[2] && st[0] + x[4] == o[8] && st[1 * Ns] + x[5] == o[9] && qf.c == o[6] &&
						qf.s == o[7];
			replayDiffs += same ? 0 : 1;
		}
	}
	if ( unsupported )
		atomicAdd( it.status + 0, unsupported );
	if ( mismatches )
		atomicAdd( it.status + 2, mismatches );
	if ( replayDiffs )
		atomicAdd( it.status + 3, replayDiffs );
}

/* ------------------------------------------------------------------ reverse */
/* What the reverse pass holds of a world: the replay of the current step (D), the body
 * adjoints and the impulse adjoints, in shared memory when the world is small. */
struct AdjReverse
{
	const float* D;
	float* adj; /* [f * Ns + b], ADJ_BODY fields */
	AdjStep L;
};

__device__ __forceinline__ Row reverse_load_row( const AdjReverse& X, int k, const b2gStepConst& sc )
{
	const int Rs = X.L.Rs;
	const float* f = X.D + X.L.rows + k;
	Row r;
	r.ia = __float_as_int( f[0] );
	r.ib = __float_as_int( f[Rs] );
	r.count = __float_as_int( f[2 * Rs] );
	r.n = gv( f[3 * Rs], f[4 * Rs] );
	r.friction = f[5 * Rs];
	r.restitution = f[6 * Rs];
	const float* soft = ( r.ia < 0 || r.ib < 0 ) ? sc.staticSoft : sc.contactSoft;
	r.biasRate = soft[0];
	r.massScale = soft[1];
	r.impulseScale = soft[2];
	r.mA = f[7 * Rs];
	r.iA = f[8 * Rs];
	r.mB = f[9 * Rs];
	r.iB = f[10 * Rs];
#pragma unroll
	for ( int j = 0; j < 2; ++j )
	{
		r.rA[j] = gv( f[( 11 + 2 * j ) * Rs], f[( 12 + 2 * j ) * Rs] );
		r.rB[j] = gv( f[( 15 + 2 * j ) * Rs], f[( 16 + 2 * j ) * Rs] );
		r.base[j] = f[( 19 + j ) * Rs];
		r.nMass[j] = f[( 21 + j ) * Rs];
		r.tMass[j] = f[( 23 + j ) * Rs];
		r.relVel[j] = f[( 25 + j ) * Rs];
		r.ni[j] = r.ti[j] = r.maxNi[j] = 0.0f;
	}
	return r;
}

__device__ __forceinline__ void get_velocity( const float* p, int Rs, DevState& A, DevState& B )
{
	A.v = gv( p[0], p[Rs] );
	A.w = p[2 * Rs];
	B.v = gv( p[3 * Rs], p[4 * Rs] );
	B.w = p[5 * Rs];
}

/* What one row of a stage needs besides its record and the adjoints. */
struct RowForward
{
	SolveForward F;	   /* solve, relax */
	DevState sa[2], sb[2]; /* restitution */
};

/* Takes it from the replay; sets the row's impulses to those before the stage. */
template <int PHASE>
__device__ __forceinline__ void reverse_forward( const AdjReverse& X, int k, Row& r, int sub, const b2gStepConst& sc, bool scalar, RowForward& f )
{
	const int Rs = X.L.Rs, Ns = X.L.Ns;
	if ( PHASE == 0 )
	{
		const float* t = X.D + X.L.warm( sub ) + k;
		r.ni[0] = t[0];
		r.ni[1] = t[Rs];
		r.ti[0] = t[2 * Rs];
		r.ti[1] = t[3 * Rs];
	}
	else if ( PHASE == 3 )
	{
		const float* t = X.D + X.L.rest() + k;
		r.ni[0] = t[0];
		r.ni[1] = t[Rs];
		r.maxNi[0] = t[2 * Rs];
		r.maxNi[1] = t[3 * Rs];
#pragma unroll
		for ( int j = 0; j < 2; ++j )
		{
			f.sa[j] = identity_state();
			f.sb[j] = identity_state();
			get_velocity( t + ( 4 + 6 * j ) * Rs, Rs, f.sa[j], f.sb[j] );
		}
	}
	else
	{
		const float* t = X.D + X.L.solve( sub, PHASE == 2 ) + k;
		const float* snap = X.D + X.L.snap + (size_t)( 2 * sub + ( PHASE == 2 ? 2 : 0 ) ) * ADJ_SNAP * Ns;
		DevState sa[4], sb[4];
		DevState A = identity_state(), B = identity_state();
		if ( r.ia >= 0 )
		{
			A.dp = gv( snap[4 * Ns + r.ia], snap[5 * Ns + r.ia] );
			A.dq = grot( snap[6 * Ns + r.ia], snap[7 * Ns + r.ia] );
		}
		if ( r.ib >= 0 )
		{
			B.dp = gv( snap[4 * Ns + r.ib], snap[5 * Ns + r.ib] );
			B.dq = grot( snap[6 * Ns + r.ib], snap[7 * Ns + r.ib] );
		}
		r.ni[0] = t[0];
		r.ni[1] = t[Rs];
		r.ti[0] = t[2 * Rs];
		r.ti[1] = t[3 * Rs];
#pragma unroll
		for ( int j = 0; j < 4; ++j )
		{
			sa[j] = A;
			sb[j] = B;
			get_velocity( t + ( 4 + 6 * j ) * Rs, Rs, sa[j], sb[j] );
		}
		solve_forward( r, sa, sb, PHASE == 1, sc, scalar, f.F );
	}
}

/* Reverse of one row of a stage (its velocity, impulse and position-delta adjoints).  The
 * scalar overflow rows share the lane rows' derivatives: the arithmetic is the same up to
 * operand grouping, a point past the manifold's count is a zero point of the lane layout,
 * and a restitution-free overflow row is skipped as the forward skipped it. */
template <int PHASE>
__device__ __forceinline__ void reverse_row( const AdjReverse& X, const Row& r, const RowForward& f, RowAdj& ra, const b2gStepConst& sc, bool scalar )
{
	if ( PHASE == 3 && scalar && r.restitution == 0.0f )
		return;
	const int Ns = X.L.Ns;
	const bool hasA = r.ia >= 0, hasB = r.ib >= 0;
	float* gA = X.adj + ( hasA ? r.ia : 0 );
	float* gB = X.adj + ( hasB ? r.ib : 0 );
	BodyV aA = { 0.0f, 0.0f, 0.0f }, aB = { 0.0f, 0.0f, 0.0f };
	float dpA[2] = { 0.0f, 0.0f }, dqA[2] = { 0.0f, 0.0f }, dpB[2] = { 0.0f, 0.0f }, dqB[2] = { 0.0f, 0.0f };
	if ( hasA )
		aA = { gA[4 * Ns], gA[5 * Ns], gA[6 * Ns] };
	if ( hasB )
		aB = { gB[4 * Ns], gB[5 * Ns], gB[6 * Ns] };
	if ( PHASE == 0 )
	{
		/* the velocities before a warm start carry the same adjoints as those after it */
		warm_vjp( r, aA, aB, ra );
		return;
	}
	if ( PHASE == 3 )
		restitution_reverse( r, f.sa, f.sb, sc, aA, aB, ra );
	else
		solve_reverse( r, f.F, aA, aB, ra, dpA, dqA, dpB, dqB );
	if ( hasA )
	{
		gA[4 * Ns] = aA.vx;
		gA[5 * Ns] = aA.vy;
		gA[6 * Ns] = aA.w;
		if ( PHASE != 3 )
		{
			gA[7 * Ns] += dpA[0];
			gA[8 * Ns] += dpA[1];
			gA[9 * Ns] += dqA[0];
			gA[10 * Ns] += dqA[1];
		}
	}
	if ( hasB )
	{
		gB[4 * Ns] = aB.vx;
		gB[5 * Ns] = aB.vy;
		gB[6 * Ns] = aB.w;
		if ( PHASE != 3 )
		{
			gB[7 * Ns] += dpB[0];
			gB[8 * Ns] += dpB[1];
			gB[9 * Ns] += dqB[0];
			gB[10 * Ns] += dqB[1];
		}
	}
}

/* Row adjoints outside registers: field f of row k at [f * Rs + k]. */
__device__ __forceinline__ RowAdj radj_load( const float* p, int Rs )
{
	RowAdj ra;
	float* o = (float*)&ra;
#pragma unroll
	for ( int i = 0; i < ADJ_RADJ; ++i )
		o[i] = p[(size_t)i * Rs];
	return ra;
}
__device__ __forceinline__ void radj_store( float* p, int Rs, const RowAdj& ra )
{
	const float* o = (const float*)&ra;
#pragma unroll
	for ( int i = 0; i < ADJ_RADJ; ++i )
		p[(size_t)i * Rs] = o[i];
}

/* Reverse of one stage: colours in reverse order, then the overflow rows in reverse
 * order.  REG: row k's record and adjoint live in lane k's registers, turn is its place
 * among the active colours (overflow rows: the number of them and up, serially). */
template <int PHASE, bool REG>
__device__ __forceinline__ void reverse_stage( const AdjReverse& X, const b2gTapeStep& h, Row mine, RowAdj& ra, int turn, int turns, float* radj,
											   int sub, const b2gStepConst& sc )
{
	const int lane = threadIdx.x, Rs = X.L.Rs;
	const int active = h.activeCount;
	if constexpr ( REG )
	{
		/* all rows at once up to their adjoints, which then pass through them in turn */
		RowForward f;
		if ( turn >= 0 )
			reverse_forward<PHASE>( X, lane, mine, sub, sc, turn >= active, f );
		if ( PHASE == 0 )
		{
			/* a warm start changes no velocity adjoint: no turns */
			if ( turn >= 0 )
				reverse_row<PHASE>( X, mine, f, ra, sc, false );
			__syncwarp();
			return;
		}
		for ( int a = active - 1; a >= 0; --a )
		{
			if ( turn == a )
				reverse_row<PHASE>( X, mine, f, ra, sc, false );
			__syncwarp();
		}
		for ( int a = turns - 1; a >= active; --a )
		{
			if ( turn == a )
				reverse_row<PHASE>( X, mine, f, ra, sc, true );
			__syncwarp();
		}
	}
	else
	{
		for ( int a = active - 1; a >= 0; --a )
		{
			const int c = h.active[a];
			for ( int k = h.colorStart[c] + lane; k < h.colorStart[c + 1]; k += ADJ_WARP )
			{
				RowForward f;
				Row r = reverse_load_row( X, k, sc );
				RowAdj g = radj_load( radj + k, Rs );
				reverse_forward<PHASE>( X, k, r, sub, sc, false, f );
				reverse_row<PHASE>( X, r, f, g, sc, false );
				radj_store( radj + k, Rs, g );
			}
			__syncwarp();
		}
		if ( lane == 0 )
		{
			for ( int k = h.colorStart[B2G_COLORS] - 1; k >= h.colorStart[B2G_OVERFLOW]; --k )
			{
				RowForward f;
				Row r = reverse_load_row( X, k, sc );
				RowAdj g = radj_load( radj + k, Rs );
				reverse_forward<PHASE>( X, k, r, sub, sc, true, f );
				reverse_row<PHASE>( X, r, f, g, sc, true );
				radj_store( radj + k, Rs, g );
			}
		}
		__syncwarp();
	}
}

/* The preparation and manifold Jacobian of one row: adjoints of both bodies' poses
 * (gpos), the velocity terms (g) and the warm-start impulses, which go to the row of the
 * step before (lamNext). */
__device__ __forceinline__ void reverse_prepare( const AdjReverse& X, int k, const Row& r, const RowAdj& ra, const b2gStepConst& sc, float* gpos,
												 b2gVec* g, float* lamNext )
{
	const int Rs = X.L.Rs, Ns = X.L.Ns;
	const float* s0 = X.D + X.L.snap; /* snapshot 0: step-start velocities */
	DevState sA = identity_state(), sB = identity_state();
	if ( r.ia >= 0 )
	{
		sA.v = gv( s0[r.ia], s0[Ns + r.ia] );
		sA.w = s0[2 * Ns + r.ia];
	}
	if ( r.ib >= 0 )
	{
		sB.v = gv( s0[r.ib], s0[Ns + r.ib] );
		sB.w = s0[2 * Ns + r.ib];
	}
	float mAdj[12], lamIn[4];
	prepare_parts( r, sA, sB, ra, sc.enableWarmStarting ? 1.0f : 0.0f, mAdj, g, lamIn );
	const float* J = X.D + X.L.jac + k;
#pragma unroll
	for ( int d = 0; d < 6; ++d )
		gpos[d] = 0.0f;
#pragma unroll
	for ( int o = 0; o < 12; ++o )
#pragma unroll
		for ( int d = 0; d < 6; ++d )
			gpos[d] += mAdj[o] * J[( o * 6 + d ) * Rs];
	const int link = __float_as_int( X.D[X.L.rows + 27 * Rs + k] );
	if ( link >= 0 )
	{
		float* lam = lamNext + ( link & 0xffffff );
#pragma unroll
		for ( int j = 0; j < 2; ++j )
		{
			const int jo = ( link >> ( 24 + 2 * j ) ) & 3;
			if ( j < r.count && jo != ADJ_LINK_NONE )
			{
				lam[(size_t)jo * Rs] += lamIn[j];
				lam[(size_t)( 2 + jo ) * Rs] += lamIn[2 + j];
			}
		}
	}
}

/* Adds a row's preparation adjoints to its bodies. */
__device__ __forceinline__ void reverse_pose( const AdjReverse& X, const Row& r, const float* gpos, const b2gVec* g )
{
	const int Ns = X.L.Ns;
	float* gA = X.adj + ( r.ia >= 0 ? r.ia : 0 );
	float* gB = X.adj + ( r.ib >= 0 ? r.ib : 0 );
	BodyV aA = { 0.0f, 0.0f, 0.0f }, aB = { 0.0f, 0.0f, 0.0f };
	if ( r.ia >= 0 )
		aA = { gA[4 * Ns], gA[5 * Ns], gA[6 * Ns] };
	if ( r.ib >= 0 )
		aB = { gB[4 * Ns], gB[5 * Ns], gB[6 * Ns] };
#pragma unroll
	for ( int j = 0; j < 2; ++j )
		if ( j < r.count )
			dv_velocities( g[j], r.rA[j], r.rB[j], aA, aB );
	if ( r.ia >= 0 )
	{
		const float* st = X.D + X.L.start + r.ia;
		gA[0 * Ns] += gpos[0];
		gA[1 * Ns] += gpos[1];
		gA[2 * Ns] += gpos[2] * -st[3 * Ns];
		gA[3 * Ns] += gpos[2] * st[2 * Ns];
		gA[4 * Ns] = aA.vx;
		gA[5 * Ns] = aA.vy;
		gA[6 * Ns] = aA.w;
	}
	if ( r.ib >= 0 )
	{
		const float* st = X.D + X.L.start + r.ib;
		gB[0 * Ns] += gpos[3];
		gB[1 * Ns] += gpos[4];
		gB[2 * Ns] += gpos[5] * -st[3 * Ns];
		gB[3 * Ns] += gpos[5] * st[2 * Ns];
		gB[4 * Ns] = aB.vx;
		gB[5 * Ns] = aB.vy;
		gB[6 * Ns] = aB.w;
	}
}

/* Shared memory of the reverse pass: two replays, body adjoints, impulse adjoints of this
 * step and the next, row adjoints unless they are in registers, step header. */
static __host__ __device__ size_t adj_reverse_floats( const AdjStep& L, bool reg )
{
	return 2 * L.copy + (size_t)ADJ_BODY * L.Ns + 8u * (size_t)L.Rs + ( reg ? 0u : (size_t)ADJ_RADJ * L.Rs );
}

/* Polls of a bulk copy's barrier before the pass gives up. */
#define ADJ_SPIN_LIMIT ( 1 << 20 )

__device__ __forceinline__ bool adj_wait( unsigned bar, unsigned parity )
{
	for ( int left = ADJ_SPIN_LIMIT; left > 0; --left )
	{
		unsigned done;
		asm volatile( "{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
					  : "=r"( done )
					  : "r"( bar ), "r"( parity )
					  : "memory" );
		if ( done )
			return true;
	}
	return false;
}

/* The reverse pass of one world over steps stepCount - 1 - first - t, t in [0, chunk).
 * SMEM: replays come to shared memory by bulk copies, one step ahead; else they are read
 * where they are.  REG: at most 32 rows, one per lane. */
template <bool SMEM, bool REG>
__global__ void __launch_bounds__( ADJ_WARP ) k_adjoint_reverse( const b2gAdjointItem* items, int first, int chunk )
{
	extern __shared__ __align__( 16 ) float sm[];
	__shared__ __align__( 8 ) unsigned long long s_bar[2];
	__shared__ b2gTapeStep s_h;
	const b2gAdjointItem& it = items[blockIdx.x];
	const int lane = threadIdx.x;
	const int N = it.bodies;
	AdjReverse X;
	X.L = adj_step( N, it.maxRows, it.maxSub );
	const int Rs = X.L.Rs, Ns = X.L.Ns;
	AdjWorld G;
	adj_world( &G, it.scratch, Ns, Rs, it.chunk );
	const int left = it.stepCount - first;
	const int n = left < chunk ? left : chunk;
	if ( n <= 0 )
		return;
	float* lam = G.lam; /* this step's */
	float* lamNext;
	float* radjShared = nullptr;
	if constexpr ( SMEM )
	{
		X.adj = sm + 2 * X.L.copy;
		lam = X.adj + ADJ_BODY * Ns;
		lamNext = lam + 4 * Rs;
		radjShared = lamNext + 4 * Rs;
	}
	else
	{
		X.adj = G.bodyAdj;
		lamNext = G.lam + 4 * Rs;
	}
	const unsigned bar = (unsigned)__cvta_generic_to_shared( s_bar );
	const unsigned buffer = (unsigned)__cvta_generic_to_shared( sm );
	const unsigned bytes = 4u * (unsigned)X.L.copy;
	auto fetch = [&]( int t ) {
		if ( lane == 0 )
		{
			const unsigned b = bar + 8u * (unsigned)( t & 1 );
			asm volatile( "mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"( b ), "r"( bytes ) : "memory" );
			asm volatile( "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
							  buffer + ( t & 1 ) * bytes ),
						  "l"( it.stepScratch + (size_t)t * it.stepFloats ), "r"( bytes ), "r"( b )
						  : "memory" );
		}
	};
	if constexpr ( SMEM )
	{
		if ( lane == 0 )
		{
			asm volatile( "mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"( bar ) : "memory" );
			asm volatile( "mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"( bar + 8u ) : "memory" );
			asm volatile( "fence.proxy.async.shared::cta;" ::: "memory" );
		}
		__syncwarp();
		fetch( 0 );
	}
	/* carried from the chunk before, or nothing yet */
	if ( SMEM || first == 0 )
	{
		for ( int i = lane; i < ADJ_BODY * Ns; i += ADJ_WARP )
			X.adj[i] = first == 0 ? 0.0f : G.bodyAdj[i];
		for ( int i = lane; i < 4 * Rs; i += ADJ_WARP )
			lam[i] = first == 0 ? 0.0f : G.lam[i];
	}
	if ( first == 0 )
		for ( int i = lane; i < 4 * N; i += ADJ_WARP )
			G.pose[i] = 0.0f;
	for ( int i = lane; i < 4 * Rs; i += ADJ_WARP )
		lamNext[i] = 0.0f;

	for ( int t = 0; t < n; ++t )
	{
		const int ts = it.stepCount - 1 - ( first + t );
		__syncwarp();
		for ( int i = lane; i < (int)( sizeof( b2gTapeStep ) / 4 ); i += ADJ_WARP )
			( (int*)&s_h )[i] = ( (const int*)( it.steps + ts ) )[i];
		if constexpr ( SMEM )
		{
			if ( t + 1 < n )
				fetch( t + 1 );
			if ( __all_sync( 0xffffffffu, adj_wait( bar + 8u * (unsigned)( t & 1 ), (unsigned)( t >> 1 ) & 1u ) ) == false )
			{
				/* the copy in flight must not outlive the shared memory it writes */
				if ( t + 1 < n )
					adj_wait( bar + 8u * (unsigned)( ( t + 1 ) & 1 ), (unsigned)( ( t + 1 ) >> 1 ) & 1u );
				if ( lane == 0 )
					atomicAdd( it.status + 3, 1 );
				return;
			}
			X.D = sm + (size_t)( t & 1 ) * X.L.copy;
		}
		else
			X.D = it.stepScratch + (size_t)t * it.stepFloats;
		__syncwarp();
		const b2gTapeStep& h = s_h;
		const b2gStepConst& sc = h.sc;
		const int R = h.rows;
		const int S = sc.subSteps;
		float* mu = G.mu + (size_t)t * Rs;
		if ( h.solve == 0 || S > ADJ_MAX_SUBSTEPS )
		{
			for ( int i = lane; i < 4 * Rs; i += ADJ_WARP )
				lam[i] = 0.0f;
			for ( int k = lane; k < Rs; k += ADJ_WARP )
				mu[k] = 0.0f;
			continue;
		}
		float* radj = SMEM ? radjShared : it.stepScratch + (size_t)t * it.stepFloats + X.L.work;

		for ( int b = lane; b < N; b += ADJ_WARP )
		{
			const float* st = X.D + X.L.start + b;
			float g[ADJ_BODY];
#pragma unroll
			for ( int i = 0; i < ADJ_BODY; ++i )
				g[i] = X.adj[i * Ns + b];
			const float* fin = X.D + X.L.snap + (size_t)2 * S * ADJ_SNAP * Ns + b;
			const float qc = st[2 * Ns], qs = st[3 * Ns], lcx = st[4 * Ns], lcy = st[5 * Ns];
			if ( st[8 * Ns] != 0.0f )
			{
				/* seed: the loss gradient with respect to the state after the last step */
				if ( ts == it.stepCount - 1 )
				{
					/* final rotation q' = normalize( dq q ) */
					b2gRot qf = gnormrot( gmulrot( grot( fin[6 * Ns], fin[7 * Ns] ), grot( qc, qs ) ) );
					const float* gf = it.gradFinal + 6 * b;
					/* p = c - rotate( q, lc ); angle: dq/dangle = ( -q.s, q.c ) */
					g[0] = gf[0];
					g[1] = gf[1];
					g[2] = gf[2] * -qf.s - ( gf[0] * lcx + gf[1] * lcy );
					g[3] = gf[2] * qf.c - ( -gf[0] * lcy + gf[1] * lcx );
					g[4] = gf[3];
					g[5] = gf[4];
					g[6] = gf[5];
				}
				/* reverse: finalisation */
				finalize_vjp( qc, qs, fin[6 * Ns], fin[7 * Ns], g );
			}
			else
			{
#pragma unroll
				for ( int i = 0; i < ADJ_BODY; ++i )
					g[i] = 0.0f;
			}
#pragma unroll
			for ( int i = 0; i < ADJ_BODY; ++i )
				X.adj[i * Ns + b] = g[i];
			float* pose = G.pose + 4 * b;
			pose[0] = qc;
			pose[1] = qs;
			pose[2] = lcx;
			pose[3] = lcy;
		}

		/* rows; stored impulses receive the next step's warm-start adjoint */
		Row mine;
		RowAdj ra;
		int turn = -1;
		const int turns = h.activeCount + h.colorStart[B2G_COLORS] - h.colorStart[B2G_OVERFLOW];
		if constexpr ( REG )
		{
			mine = reverse_load_row( X, lane < R ? lane : 0, sc );
			ra = RowAdj{};
			for ( int a = 0; a < h.activeCount; ++a )
				if ( lane >= h.colorStart[h.active[a]] && lane < h.colorStart[h.active[a] + 1] )
					turn = a;
			if ( lane >= h.colorStart[B2G_OVERFLOW] && lane < R )
				turn = h.activeCount + lane - h.colorStart[B2G_OVERFLOW];
			if ( lane < R )
			{
				ra.ni[0] += lam[lane];
				ra.ni[1] += lam[Rs + lane];
				ra.ti[0] += lam[2 * Rs + lane];
				ra.ti[1] += lam[3 * Rs + lane];
			}
		}
		else
		{
			for ( int k = lane; k < R; k += ADJ_WARP )
			{
				RowAdj g{};
				g.ni[0] += lam[k];
				g.ni[1] += lam[Rs + k];
				g.ti[0] += lam[2 * Rs + k];
				g.ti[1] += lam[3 * Rs + k];
				radj_store( radj + k, Rs, g );
			}
		}
		__syncwarp();

		/* reverse: restitution, then the substeps */
		reverse_stage<3, REG>( X, h, mine, ra, turn, turns, radj, 0, sc );
		for ( int sub = S - 1; sub >= 0; --sub )
		{
			reverse_stage<2, REG>( X, h, mine, ra, turn, turns, radj, sub, sc );
			for ( int b = lane; b < N; b += ADJ_WARP )
			{
				if ( X.D[X.L.start + 8 * Ns + b] == 0.0f )
					continue;
				const float* s = X.D + X.L.snap + (size_t)( 2 * sub + 1 ) * ADJ_SNAP * Ns + b;
				float pre[8] = { 0.0f, 0.0f, s[2 * Ns], 0.0f, 0.0f, 0.0f, s[6 * Ns], s[7 * Ns] };
				float g[ADJ_BODY];
#pragma unroll
				for ( int i = 4; i < 11; ++i )
					g[i] = X.adj[i * Ns + b];
				ip_vjp( pre, sc.h, g );
#pragma unroll
				for ( int i = 4; i < 11; ++i )
					X.adj[i * Ns + b] = g[i];
			}
			__syncwarp();
			reverse_stage<1, REG>( X, h, mine, ra, turn, turns, radj, sub, sc );
			if ( sc.enableWarmStarting )
				reverse_stage<0, REG>( X, h, mine, ra, turn, turns, radj, sub, sc );
			for ( int b = lane; b < N; b += ADJ_WARP )
			{
				if ( X.D[X.L.start + 8 * Ns + b] == 0.0f )
					continue;
				const float* s = X.D + X.L.snap + (size_t)( 2 * sub ) * ADJ_SNAP * Ns + b;
				const float* tm = X.D + X.L.terms + b;
				float pre[3] = { s[0], s[Ns], s[2 * Ns] };
				float g[ADJ_BODY];
#pragma unroll
				for ( int i = 4; i < 7; ++i )
					g[i] = X.adj[i * Ns + b];
				iv_vjp( pre, make_float4( tm[0], tm[Ns], tm[2 * Ns], tm[3 * Ns] ), tm[4 * Ns], sc, g );
#pragma unroll
				for ( int i = 4; i < 7; ++i )
					X.adj[i * Ns + b] = g[i];
			}
			__syncwarp();
		}

		/* reverse: preparation and the manifold Jacobian; the bodies' sums colour by colour
		 * so that no two lanes update one body, then the overflow rows in order */
		if constexpr ( REG )
		{
			float gpos[6];
			b2gVec g[2];
			if ( lane < R )
			{
				reverse_prepare( X, lane, mine, ra, sc, gpos, g, lamNext );
				mu[lane] = ra.mu;
			}
			for ( int a = 0; a < turns; ++a )
			{
				if ( turn == a )
					reverse_pose( X, mine, gpos, g );
				__syncwarp();
			}
		}
		else
		{
			for ( int a = 0; a <= h.activeCount; ++a )
			{
				const bool ov = a == h.activeCount;
				const int c = ov ? B2G_OVERFLOW : h.active[a];
				const int lo = ov ? ( lane == 0 ? h.colorStart[c] : h.colorStart[c + 1] ) : h.colorStart[c] + lane;
				for ( int k = lo; k < h.colorStart[c + 1]; k += ov ? 1 : ADJ_WARP )
				{
					float gpos[6];
					b2gVec g[2];
					const Row r = reverse_load_row( X, k, sc );
					const RowAdj ga = radj_load( radj + k, Rs );
					reverse_prepare( X, k, r, ga, sc, gpos, g, lamNext );
					mu[k] = ga.mu;
					reverse_pose( X, r, gpos, g );
				}
				__syncwarp();
			}
		}
		for ( int k = R + lane; k < Rs; k += ADJ_WARP )
			mu[k] = 0.0f;
		/* position deltas start each step at zero: their adjoints end here */
		for ( int b = lane; b < N; b += ADJ_WARP )
		{
#pragma unroll
			for ( int i = 7; i < 11; ++i )
				X.adj[i * Ns + b] = 0.0f;
		}
		/* the impulse adjoints collected for the step before are its own now */
		for ( int i = lane; i < 4 * Rs; i += ADJ_WARP )
		{
			lam[i] = lamNext[i];
			lamNext[i] = 0.0f;
		}
	}
	__syncwarp();

	if ( SMEM )
	{
		for ( int i = lane; i < ADJ_BODY * Ns; i += ADJ_WARP )
			G.bodyAdj[i] = X.adj[i];
		for ( int i = lane; i < 4 * Rs; i += ADJ_WARP )
			G.lam[i] = lam[i];
	}
	if ( first + n < it.stepCount )
		return;
	/* gradient with respect to the state at the start of the first recorded step:
	 * p = c - rotate( q, lc ), angle with dq/dangle = ( -q.s, q.c ) */
	for ( int b = lane; b < N; b += ADJ_WARP )
	{
		const float* pose = G.pose + 4 * b;
		const float* g = X.adj + b;
		float* out = it.gradInitial + 6 * b;
		float qc = pose[0], qs = pose[1], lcx = pose[2], lcy = pose[3];
		out[0] = g[0];
		out[1] = g[Ns];
		out[2] = g[2 * Ns] * -qs + g[3 * Ns] * qc + g[0] * ( -qs * lcx - qc * lcy ) + g[Ns] * ( qc * lcx - qs * lcy );
		out[3] = g[4 * Ns];
		out[4] = g[5 * Ns];
		out[5] = g[6 * Ns];
	}
	if ( lane == 0 )
		it.status[1] = it.status[2] + it.status[3];
}

/* Friction gradient of the chunk's rows, mu_row = sqrt( muA muB ): one thread per shape
 * adds the rows that touch it, the last step's first, rows in order.  Rows are taken
 * ADJ_FRICTION at a time through shared memory. */
#define ADJ_FRICTION 256

__global__ void __launch_bounds__( ADJ_FRICTION ) k_adjoint_friction( const b2gAdjointItem* items, int first, int chunk )
{
	const b2gAdjointItem& it = items[blockIdx.x];
	const AdjStep L = adj_step( it.bodies, it.maxRows, it.maxSub );
	AdjWorld G;
	adj_world( &G, it.scratch, L.Ns, L.Rs, it.chunk );
	const int left = it.stepCount - first;
	const int n = left < chunk ? left : chunk;
	const int tid = threadIdx.x;
	__shared__ int2 shape[ADJ_FRICTION];
	__shared__ float2 part[ADJ_FRICTION];
	const int total = n > 0 ? n * L.Rs : 0;
	for ( int s0 = 0; s0 < it.shapes; s0 += ADJ_FRICTION )
	{
		const int s = s0 + tid;
		float sum = s < it.shapes && first > 0 ? it.gradFriction[s] : 0.0f;
		for ( int e0 = 0; e0 < total; e0 += ADJ_FRICTION )
		{
			const int e = e0 + tid;
			int2 who = make_int2( -1, -1 );
			float2 add = make_float2( 0.0f, 0.0f );
			if ( e < total )
			{
				const int t = e / L.Rs, k = e - t * L.Rs;
				const float gmu = G.mu[e];
				if ( gmu != 0.0f )
				{
					const b2gTapeRow& tr = it.tapeRows[it.steps[it.stepCount - 1 - ( first + t )].rowOff + k];
					float muA = it.shapeFriction[tr.shapeA], muB = it.shapeFriction[tr.shapeB];
					if ( muA > 0.0f )
					{
						who.x = tr.shapeA;
						add.x = gmu * 0.5f * tr.friction / muA;
					}
					if ( muB > 0.0f )
					{
						who.y = tr.shapeB;
						add.y = gmu * 0.5f * tr.friction / muB;
					}
				}
			}
			shape[tid] = who;
			part[tid] = add;
			__syncthreads();
			const int m = total - e0 < ADJ_FRICTION ? total - e0 : ADJ_FRICTION;
			for ( int i = 0; i < m; ++i )
			{
				if ( shape[i].x == s )
					sum += part[i].x;
				if ( shape[i].y == s )
					sum += part[i].y;
			}
			__syncthreads();
		}
		if ( s < it.shapes )
			it.gradFriction[s] = sum;
	}
}

/* The backward pass of `count` worlds (device item array), `steps` the most recorded
 * steps of one, `chunk` steps at a time: one replay, one reverse and one friction launch
 * each.  bodies, rows, subSteps: the largest of the worlds. */
extern "C" int b2gd_adjoint_launch( const b2gAdjointItem* dItems, int count, int steps, int chunk, int bodies, int rows, int subSteps, void* stream )
{
	if ( count <= 0 )
		return 0;
	cudaStream_t s = (cudaStream_t)stream;
	const AdjStep L = adj_step( bodies, at_least_one( rows ), subSteps );
	const bool reg = rows <= ADJ_WARP;
	const size_t bytes = 4u * adj_reverse_floats( L, reg );
	const bool smem = bytes <= 220u * 1024u;
	auto kernel = smem ? ( reg ? k_adjoint_reverse<true, true> : k_adjoint_reverse<true, false> ) : k_adjoint_reverse<false, false>;
	if ( smem )
	{
		cudaError_t e = cudaFuncSetAttribute( kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024 );
		if ( e != cudaSuccess )
			return (int)e;
	}
	for ( int first = 0; first < steps; first += chunk )
	{
		const int n = steps - first < chunk ? steps - first : chunk;
		/* in one dimension of the grid, the only one for more than 65535 worlds or steps */
		k_adjoint_replay<<<(unsigned)n * (unsigned)count, ADJ_WARP, 0, s>>>( dItems, first, n );
		kernel<<<count, ADJ_WARP, smem ? bytes : 0, s>>>( dItems, first, n );
		k_adjoint_friction<<<count, ADJ_FRICTION, 0, s>>>( dItems, first, n );
	}
	return (int)cudaGetLastError();
}
