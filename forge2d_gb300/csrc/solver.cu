// Soft-step solver of the world step, GPU-first.
//
// Stage order is that of b2SolverTask (packages/forge2d/third_party/box2d/
// src/solver.c:929-1160): prepare joints and contacts; per substep integrate
// velocities, warm start (overflow joints, overflow contacts, then graph
// colours 0..10), solve, integrate positions, relax; then restitution and
// impulse storage. After the set-up launches all of it runs in one persistent
// launch in which no stage waits for the whole device: the constraints are a
// data flow over the bodies (k_solve).
#include "dscan.cuh"
#include "dsync.cuh"

#include "dsolve.cuh"
#include "dworld.cuh"
#include "joint.cuh"
#include "kernels.cuh"

struct SolveParams
{
	float h, inv_h, dt, inv_dt;
	Soft contactSoft, staticSoft, jointSoft;
	float minBiasVel; // -contactSpeed (world.c:767)
	float pushout;	  // maxContactPushSpeed (overflow path)
	float restitutionThreshold;
	float maxLinearSpeed, maxAngularSpeed;
	fv2 gravity;
	int subSteps;	 // of this launch
	int restitution; // this launch ends the step: restitution and impulse storage
	int enableWarmStarting;
	int parts;	  // blocks of the solver launch
	int minChunk; // bodies per part, at least
	int onePart;  // up to this many bodies with constraints make one part
	int slots;	  // bodies whose rows fit a block's shared memory
};

#define FLOW_SENTINEL 0xffffffffu
// Overflow constraints of one body whose ranks are found by walking its list,
// and of one part that are ordered by counting, at most: both are quadratic,
// but their threads run together. Longer ones are ranked in one pass over all
// overflow constraints (flow_rank_long).
#define FLOW_WALK 256
#define FLOW_SORT 1024
// Polls without progress before a warp gives up. A warp may rightly wait for a
// whole stage's chain of one body's overflow constraints (0.8 us each, up to
// 15 polls), so they count towards it.
#define FLOW_SPIN_LIMIT ( 1 << 22 )
#define FLOW_SPIN_OVERFLOW 256
#define FLOW_OVERFLOW_MOST ( 1 << 21 )
#define FLOW_REST_SHIFT 11		  // bodyOrd.x: colour bits, then the bits of colours with restitution,
#define FLOW_GLOBAL ( 1 << 22 )	  // and whether the body's row is shared between blocks
#define FLOW_COLOURS ( ( 1 << F2D_OVERFLOW ) - 1 )
#define BI_AWAKE 1 // bodyInt flags
#define BI_FAST_ROT 2

__device__ __forceinline__ bool body_awake( int f )
{
	return ( f & ( BF_USED | BF_ENABLED | BF_ASLEEP ) ) == ( BF_USED | BF_ENABLED ) && body_type( f ) != 0;
}

// ---------------------------------------------------------------------------
// parts: bodies in spatial order, dealt to the solver's blocks in runs
// ---------------------------------------------------------------------------

// Position of every body with graph constraints (as of the last step's
// colours) in the order of the broadphase tree's leaves, which follow a
// Morton curve: one launch, tiles chained by decoupled look-back. bodyPos is
// the position, or -2 - position for a body without constraints, which gets no
// place of its own. The order only decides where a constraint is solved,
// never what it computes.
#define ORDER_THREADS 1024
#define ORDER_ITEMS 4
#define ORDER_TILE ( ORDER_THREADS * ORDER_ITEMS )
__global__ void __launch_bounds__( ORDER_THREADS ) k_body_order( DWorld w )
{
	__shared__ int smem[32];
	__shared__ int s_tile, s_prefix;
	const int n = w.sc->treeLeafCount;
	unsigned long long* state = w.orderState;
	if ( threadIdx.x == 0 )
		s_tile = (int)atomicAdd( (unsigned*)state, 1u );
	__syncthreads();
	const int tile = s_tile;
	const int base = tile * ORDER_TILE;
	if ( base >= n )
	{
		if ( tile == 0 && threadIdx.x == 0 )
			w.sc->orderTotal = 0;
		return;
	}
	int body[ORDER_ITEMS], flag[ORDER_ITEMS];
	int sum = 0;
#pragma unroll
	for ( int k = 0; k < ORDER_ITEMS; ++k )
	{
		int i = base + threadIdx.x * ORDER_ITEMS + k;
		body[k] = -1;
		flag[k] = 0;
		if ( i < n )
		{
			int s = w.leafShape[i];
			int b = w.shapeBody[s];
			if ( w.headShape[b] == s )
			{
				body[k] = b;
				flag[k] = w.colorMask[b] != 0u ? 1 : 0;
			}
		}
		sum += flag[k];
	}
	int aggregate;
	int excl = block_exclusive_scan_1024( sum, smem, &aggregate );
	if ( threadIdx.x == 0 )
	{
		const unsigned long long AGG = 1ull, PREFIX = 2ull;
		int prefix = 0;
		if ( tile > 0 )
		{
			st_release_u64( state + 1 + tile, ( AGG << 32 ) | (unsigned)aggregate );
			long long spins = 0;
			for ( int j = tile - 1; j >= 0; )
			{
				unsigned long long v = ld_acquire_u64( state + 1 + j );
				if ( ( v >> 32 ) == 0ull )
				{
					if ( ++spins > F2D_SPIN_LIMIT )
					{
						atomicOr( &w.sc->error, ERR_BARRIER_TIMEOUT );
						break;
					}
					continue;
				}
				prefix += (int)(unsigned)( v & 0xffffffffull );
				if ( ( v >> 32 ) == PREFIX )
					break;
				j -= 1;
			}
		}
		st_release_u64( state + 1 + tile, ( PREFIX << 32 ) | (unsigned)( prefix + aggregate ) );
		s_prefix = prefix;
		if ( base + ORDER_TILE >= n )
			w.sc->orderTotal = prefix + aggregate;
	}
	__syncthreads();
	excl += s_prefix;
#pragma unroll
	for ( int k = 0; k < ORDER_ITEMS; ++k )
	{
		if ( body[k] >= 0 )
			w.bodyPos[body[k]] = flag[k] ? excl : -2 - excl;
		if ( flag[k] )
			w.bodyAt[excl] = body[k];
		excl += flag[k];
	}
}

// Bodies per part: positions are dealt to the blocks in runs of this length.
__device__ __forceinline__ int part_chunk( const DWorld& w, const SolveParams& p )
{
	int n = w.sc->orderTotal;
	int chunk = max( p.minChunk, ( n + p.parts - 1 ) / p.parts );
	return max( n <= p.onePart ? n : chunk, 1 );
}

__device__ __forceinline__ int body_part( const DWorld& w, const SolveParams& p, int chunk, int b )
{
	int pos = w.bodyPos[b];
	pos = pos >= 0 ? pos : -2 - pos;
	return min( max( pos, 0 ) / chunk, p.parts - 1 );
}

// Part of the constraint between two bodies (-1 static): the lower of the
// bodies' parts, so that of two neighbouring parts only the higher one's
// bodies are shared. Shared bodies are marked.
__device__ __forceinline__ int constraint_part( const DWorld& w, const SolveParams& p, int chunk, int a, int b )
{
	int pa = a >= 0 ? body_part( w, p, chunk, a ) : 0x7fffffff;
	int pb = b >= 0 ? body_part( w, p, chunk, b ) : 0x7fffffff;
	int part = min( min( pa, pb ), p.parts - 1 );
	if ( a >= 0 && pa != part )
		atomicOr( (int*)( w.bodyOrd + a ), FLOW_GLOBAL );
	if ( b >= 0 && pb != part )
		atomicOr( (int*)( w.bodyOrd + b ), FLOW_GLOBAL );
	return part;
}

__device__ __forceinline__ int dynamic_index( const DWorld& w, int b )
{
	return body_type( w.bflags[b] ) == 0 ? -1 : b;
}

// Counts an overflow constraint on its bodies (a body at both its ends once)
// and returns its place in its part.
__device__ __forceinline__ int overflow_place( const DWorld& w, int part, int a, int b )
{
	if ( a >= 0 && atomicAdd( (int*)( w.bodyOrd + a ) + 1, 1 ) == FLOW_WALK )
		*w.flowLong = 1;
	if ( b >= 0 && b != a && atomicAdd( (int*)( w.bodyOrd + b ) + 1, 1 ) == FLOW_WALK )
		*w.flowLong = 1;
	int at = atomicAdd( w.binOverflow + part, 1 );
	if ( at == FLOW_SORT )
		*w.flowLong = 1;
	return at;
}

// Counts the constraints per part and colour and gives each its place there;
// per body, the factors of a substep's velocity integration (solver.c:65-130;
// they are the same in every substep).
__global__ void k_solver_count( DWorld w, SolveParams p )
{
	const int tid = blockIdx.x * blockDim.x + threadIdx.x, stride = gridDim.x * blockDim.x;
	const int chunk = part_chunk( w, p );
	const int nc = w.sc->contactIdCount;
	for ( int c = tid; c < nc; c += stride )
	{
		int col = w.ccolor[c];
		if ( col < 0 || ( w.cflags[c] & CF_USED ) == 0 )
			continue;
		int2 bd = w.cbody[c];
		const int ia = dynamic_index( w, bd.x ), ib = dynamic_index( w, bd.y );
		int part = constraint_part( w, p, chunk, ia, ib );
		if ( col < F2D_OVERFLOW )
		{
			int bin = part * F2D_OVERFLOW + col;
			w.slotPlace[c] = make_int2( bin, atomicAdd( w.binContacts + bin, 1 ) );
		}
		else
			w.slotPlace[c] = make_int2( part, overflow_place( w, part, ia, ib ) );
	}
	for ( int j = tid; j < w.jointCount; j += stride )
	{
		int col = w.jcolor[j];
		if ( ( w.jflags[j] & JF_USED ) == 0 || col < 0 )
			continue;
		int2 bd = w.jbody[j];
		const int ia = dynamic_index( w, bd.x ), ib = dynamic_index( w, bd.y );
		int part = constraint_part( w, p, chunk, ia, ib );
		if ( col < F2D_OVERFLOW )
		{
			int bin = part * F2D_OVERFLOW + col;
			w.jointPlace[j] = make_int2( bin, atomicAdd( w.binJoints + bin, 1 ) );
		}
		else
			w.jointPlace[j] = make_int2( part, overflow_place( w, part, ia, ib ) );
	}
	for ( int b = tid; b < w.bodyCount; b += stride )
	{
		float4 m = w.massv[b];
		float4 dmp = w.damp[b];
		float4 f = w.force[b];
		int flags = w.bflags[b];
		float h = p.h;
		float linearDamping = 1.0f / ( 1.0f + h * dmp.x );
		float angularDamping = 1.0f / ( 1.0f + h * dmp.y );
		float gravityScale = m.x > 0.0f ? dmp.z : 0.0f;
		fv2 g = p.gravity;
		if ( w.subCount > 0 )
		{
			float2 gb = w.bodyGravity[b];
			g = mk( gb.x, gb.y );
		}
		fv2 lvd = vadd( vscale( h * m.x, mk( f.x, f.y ) ), vscale( h * gravityScale, g ) );
		float avd = h * m.y * f.z;
		int bits = ( body_awake( flags ) ? BI_AWAKE : 0 ) | ( ( flags & BF_FAST_ROT ) ? BI_FAST_ROT : 0 );
		w.bodyInt[2 * (size_t)b] = make_float4( lvd.x, lvd.y, linearDamping, avd );
		w.bodyInt[2 * (size_t)b + 1] = make_float4( angularDamping, __int_as_float( bits ), 0.0f, 0.0f );
		// the solver counts a body's operations in its row's last word
		if ( __float_as_int( w.vel[b].w ) != 0 )
			w.vel[b].w = 0.0f;
	}
}

// Exclusive prefix over n bins in shared memory (256 threads): plain counts,
// or groups of 32.
__device__ __forceinline__ int bin_prefix( const int* bins, int n, int* out, bool groups, int* smem )
{
	int per = ( n + 255 ) / 256;
	int lo = threadIdx.x * per, hi = min( lo + per, n );
	int sum = 0;
	for ( int i = lo; i < hi; ++i )
	{
		int v = bins[i];
		sum += groups ? ( v + 31 ) >> 5 : v;
	}
	int total;
	int at = block_exclusive_scan_1024( sum, smem, &total );
	for ( int i = lo; i < hi; ++i )
	{
		out[i] = at;
		int v = bins[i];
		at += groups ? ( v + 31 ) >> 5 : v;
	}
	__syncthreads();
	return total;
}

// Notes a constraint on a body, for the ranks of the solver's data flow: its
// colour, or overflow constraint `e` (its place in the serial order: joints,
// then contacts) in the body's list.
__device__ __forceinline__ void flow_note( const DWorld& w, int b, int colour, int e, int side, bool restitution )
{
	if ( b < 0 )
		return;
	int* o = (int*)( w.bodyOrd + b );
	if ( colour < F2D_OVERFLOW )
	{
		atomicOr( o, ( 1 << colour ) | ( restitution ? 1 << ( FLOW_REST_SHIFT + colour ) : 0 ) );
		return;
	}
	if ( restitution )
		atomicAdd( o + 2, 1 );
	// list heads are keys + 1, 0 when empty
	w.ovfNext[2 * (size_t)e + side] = atomicExch( o + 3, ( ( e << 2 ) | ( restitution ? 2 : 0 ) | side ) + 1 );
}

// Bodies of overflow constraint e (-1 static), its part, and whether it has
// restitution.
__device__ __forceinline__ int4 overflow_constraint( const DWorld& w, int e, int novfJ )
{
	if ( e < novfJ )
	{
		const int j = w.overflowJoints[e];
		const int2 bd = w.jbody[j];
		return make_int4( dynamic_index( w, bd.x ), dynamic_index( w, bd.y ), w.jointPlace[j].x, 0 );
	}
	const int c = w.overflowList[e - novfJ];
	const int2 bd = w.cbody[c];
	return make_int4( dynamic_index( w, bd.x ), dynamic_index( w, bd.y ), w.slotPlace[c].x, w.cmat[c].y != 0.0f ? 1 : 0 );
}

// Ranks of overflow constraints on bodies that have more than FLOW_WALK, and
// the serial order of parts that have more than FLOW_SORT: one warp each over
// all of them in order (70 ns a constraint, bound by four dependent reads for
// 16 of them; each of the body's operations that follow, one after another in
// every stage, takes 0.8 us: 8000 circles on a plank, 0.6 of 76 ms). Walks
// between the operations made 500 circles 6.3 ms instead of 5.1 and grew with
// the square. The body's running counts stand in the free words of its bodyInt
// row.
__device__ void flow_rank_long( const DWorld& w, int novfJ, int n, int* partAt )
{
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
	const unsigned below = ( 1u << lane ) - 1u;
	if ( warp == 0 )
		for ( int base = 0; base < n; base += 16 )
		{
			const int e = base + ( lane >> 1 ), side = lane & 1;
			int key = -1 - lane, rest = 0;
			bool both = false;
			if ( e < n )
			{
				const int4 k = overflow_constraint( w, e, novfJ );
				const int b = side ? k.y : k.x;
				both = k.x == k.y;
				rest = k.w;
				if ( b >= 0 && !( both && side ) && w.bodyOrd[b].y > FLOW_WALK )
					key = b;
			}
			const unsigned rests = __ballot_sync( 0xffffffffu, rest != 0 );
			const unsigned peers = __match_any_sync( 0xffffffffu, key );
			if ( key >= 0 )
			{
				int* at = (int*)( w.bodyInt + 2 * (size_t)key + 1 ) + 2;
				const int all = __ldcg( at ) + __popc( peers & below ), some = __ldcg( at + 1 ) + __popc( peers & rests & below );
				int* r = (int*)( w.ovfRank + e );
				r[side] = all;
				r[2 + side] = some;
				if ( both )
				{
					r[1] = all;
					r[3] = some;
				}
				__syncwarp( peers );
				if ( ( peers & ~below ) == ( 1u << lane ) ) // the last of them
				{
					__stcg( at, all + 1 );
					__stcg( at + 1, some + rest );
				}
			}
			__syncwarp();
		}
	else if ( warp == 1 )
		for ( int base = 0; base < n; base += 32 )
		{
			const int e = base + lane;
			int part = -1 - lane;
			if ( e < n )
			{
				const int k = overflow_constraint( w, e, novfJ ).z;
				if ( w.binOverflow[k] > FLOW_SORT )
					part = k;
			}
			const unsigned peers = __match_any_sync( 0xffffffffu, part );
			if ( part >= 0 )
			{
				const int at = partAt[part] + __popc( peers & below );
				w.ovfSorted[at] = e;
				__syncwarp( peers );
				if ( ( peers & ~below ) == ( 1u << lane ) )
					partAt[part] = at + 1;
			}
			__syncwarp();
		}
}

// Constraint rows of every contact in the graph (contact_solver.c:1438-1669
// and :24-156, identical expressions in both), grouped by part and colour,
// overflow contacts first in overflow-array order; the joints' lists.
__global__ void __launch_bounds__( 256 ) k_solver_prepare( DWorld w, SolveParams p )
{
	extern __shared__ int dynBins[];
	__shared__ int smem[32];
	const int bins = p.parts * F2D_OVERFLOW;
	int* sContact = dynBins;
	int* sJoint = dynBins + bins;
	int* sOverflow = dynBins + 2 * bins;
	const int novf = w.sc->overflowCount, novfJ = w.sc->overflowJointCount;
	const int tid = blockIdx.x * blockDim.x + threadIdx.x, stride = gridDim.x * blockDim.x;
	bin_prefix( w.binContacts, bins, sContact, true, smem );
	if ( w.jointCount > 0 )
		bin_prefix( w.binJoints, bins, sJoint, false, smem );
	if ( novf + novfJ > 0 )
		bin_prefix( w.binOverflow, p.parts, sOverflow, false, smem );
	const int firstGroup = ( novf + 31 ) >> 5;
	if ( blockIdx.x == 0 )
	{
		// the bins' starts for the solver, and the colours' sizes
		__shared__ int colour[F2D_OVERFLOW];
		if ( threadIdx.x < F2D_OVERFLOW )
			colour[threadIdx.x] = 0;
		__syncthreads();
		for ( int i = threadIdx.x; i < bins; i += blockDim.x )
		{
			w.binContactStart[i] = firstGroup + sContact[i];
			if ( w.jointCount > 0 )
				w.binJointStart[i] = sJoint[i];
			atomicAdd( colour + i % F2D_OVERFLOW, w.binContacts[i] );
		}
		if ( novf + novfJ > 0 )
			for ( int i = threadIdx.x; i < p.parts; i += blockDim.x )
				w.binOverflowStart[i] = sOverflow[i];
		__syncthreads();
		if ( threadIdx.x == 0 )
		{
			int total = novf;
			for ( int c = 0; c < F2D_OVERFLOW; ++c )
			{
				w.sc->colorCount[c] = colour[c];
				total += colour[c];
			}
			w.sc->colorCount[F2D_OVERFLOW] = novf;
			w.sc->touchingCount = total;
		}
	}
	// joints: the solver's lists (their rows are prepared by joint.cu)
	for ( int j = tid; j < w.jointCount; j += stride )
	{
		int col = w.jcolor[j];
		if ( ( w.jflags[j] & JF_USED ) == 0 || col < 0 || col >= F2D_OVERFLOW )
			continue;
		int2 pl = w.jointPlace[j];
		w.jointSlots[sJoint[pl.x] + pl.y] = j;
		int2 bd = w.jbody[j];
		flow_note( w, dynamic_index( w, bd.x ), col, 0, 0, false );
		flow_note( w, dynamic_index( w, bd.y ), col, 0, 1, false );
	}
	for ( int e = tid; e < novfJ; e += stride )
	{
		int j = w.overflowJoints[e];
		int2 pl = w.jointPlace[j];
		w.ovfItems[sOverflow[pl.x] + pl.y] = e;
		int2 bd = w.jbody[j];
		flow_note( w, dynamic_index( w, bd.x ), F2D_OVERFLOW, e, 0, false );
		if ( bd.y != bd.x ) // a body lists a joint at both its ends once
			flow_note( w, dynamic_index( w, bd.y ), F2D_OVERFLOW, e, 1, false );
	}
	float warmStartScale = p.enableWarmStarting ? 1.0f : 0.0f;
	const int nc = w.sc->contactIdCount;
	for ( int c = tid; c < nc; c += stride )
	{
		const int col = w.ccolor[c];
		if ( col < 0 || ( w.cflags[c] & CF_USED ) == 0 )
			continue;
		int2 pl = w.slotPlace[c];
		int k;
		if ( col < F2D_OVERFLOW )
			k = 32 * ( firstGroup + sContact[pl.x] ) + pl.y;
		else
		{
			k = w.coverflowIndex[c];
			w.ovfItems[sOverflow[pl.x] + pl.y] = novfJ + k;
		}
		if ( k < 0 || k >= w.slotCap )
		{
			atomicOr( &w.sc->error, ERR_CONTACT_CAPACITY );
			continue;
		}
		int2 bd = w.cbody[c];
		int ia = dynamic_index( w, bd.x );
		int ib = dynamic_index( w, bd.y );
		float4 cm = w.cmass[c];
		float mA = cm.x, iA = cm.y, mB = cm.z, iB = cm.w;
		// constraint_graph.c:139-181: a static side carries zero mass
		if ( ia < 0 )
		{
			mA = 0.0f;
			iA = 0.0f;
		}
		if ( ib < 0 )
		{
			mB = 0.0f;
			iB = 0.0f;
		}
		fv2 vA = mk( 0.0f, 0.0f ), vB = mk( 0.0f, 0.0f );
		float wA = 0.0f, wB = 0.0f;
		if ( ia >= 0 )
		{
			float4 v = w.vel[ia];
			vA = mk( v.x, v.y );
			wA = v.z;
		}
		if ( ib >= 0 )
		{
			float4 v = w.vel[ib];
			vB = mk( v.x, v.y );
			wB = v.z;
		}
		float kk = iA + iB;
		float rollingMass = kk > 0.0f ? 1.0f / kk : 0.0f;
		float4 mn = w.mnorm[c];
		fv2 normal = mk( mn.x, mn.y );
		int pointCount = __float_as_int( mn.w );
		float4 cmat = w.cmat[c];
		flow_note( w, ia, col, novfJ + k, 0, cmat.y != 0.0f );
		flow_note( w, ib, col, novfJ + k, 1, cmat.y != 0.0f );
		float4* row = krow( w, k, 0 );
		row[32 * KR_HEAD] = make_float4( __int_as_float( ia ), __int_as_float( ib ), __int_as_float( c ),
										 __int_as_float( pointCount ) );
		row[32 * KR_MASS] = make_float4( mA, iA, mB, iB );
		row[32 * KR_NORMAL] = make_float4( normal.x, normal.y, cmat.x, cmat.w );
		row[32 * KR_MISC] = make_float4( cmat.y, cmat.z, rollingMass, warmStartScale * mn.z );
		fv2 tangent = vright( normal );
		float4 anch[2], pp[2];
		float ni[2], ti[2];
		for ( int j = 0; j < 2; ++j )
		{
			if ( j >= pointCount )
			{
				anch[j] = make_float4( 0.0f, 0.0f, 0.0f, 0.0f );
				pp[j] = make_float4( 0.0f, 0.0f, 0.0f, 0.0f );
				ni[j] = 0.0f;
				ti[j] = 0.0f;
				continue;
			}
			float4 a = w.mpA[2 * c + j];
			float4 b = w.mpB[2 * c + j];
			float4 im = w.mpI[2 * c + j];
			fv2 rA = mk( a.x, a.y ), rB = mk( a.z, a.w );
			anch[j] = a;
			float baseSeparation = b.z - vdot( vsub( rB, rA ), normal );
			ni[j] = warmStartScale * im.x;
			ti[j] = warmStartScale * im.y;
			float rnA = vcross( rA, normal );
			float rnB = vcross( rB, normal );
			float kNormal = mA + mB + iA * rnA * rnA + iB * rnB * rnB;
			float normalMass = kNormal > 0.0f ? 1.0f / kNormal : 0.0f;
			float rtA = vcross( rA, tangent );
			float rtB = vcross( rB, tangent );
			float kTangent = mA + mB + iA * rtA * rtA + iB * rtB * rtB;
			float tangentMass = kTangent > 0.0f ? 1.0f / kTangent : 0.0f;
			fv2 vrA = vadd( vA, vcrossSV( wA, rA ) );
			fv2 vrB = vadd( vB, vcrossSV( wB, rB ) );
			float relVel = vdot( normal, vsub( vrB, vrA ) );
			pp[j] = make_float4( baseSeparation, normalMass, tangentMass, relVel );
			// learned warm start: features of a point that has no cached impulse
			if ( w.learnMode != 0 && ( ( float_to_bits( b.w ) >> 16 ) & 1 ) == 0 )
			{
				int q = atomicAdd( &w.sc->newPointCount, 1 );
				if ( q < w.newPointCap )
				{
					w.newPoint[q] = make_int2( k, j );
					float* f = w.newFeat + 12 * (size_t)q;
					f[0] = normal.x;
					f[1] = normal.y;
					f[2] = relVel;
					f[3] = vdot( tangent, vsub( vrB, vrA ) );
					f[4] = b.z;
					f[5] = vdot( rA, tangent );
					f[6] = vdot( rB, tangent );
					f[7] = vdot( rA, normal );
					f[8] = vdot( rB, normal );
					f[9] = normalMass;
					f[10] = tangentMass;
					f[11] = cmat.x;
				}
			}
		}
		row[32 * KR_ANCH1] = anch[0];
		row[32 * KR_ANCH2] = anch[1];
		row[32 * KR_P1] = pp[0];
		row[32 * KR_P2] = pp[1];
		row[32 * KR_IMP] = make_float4( ni[0], ni[1], ti[0], ti[1] );
		row[32 * KR_TOT] = make_float4( 0.0f, 0.0f, 0.0f, 0.0f );
	}
	// a body or a part with many overflow constraints (counted by the launch before)
	if ( blockIdx.x == gridDim.x - 1 && *w.flowLong )
	{
		__syncthreads();
		flow_rank_long( w, novfJ, novf + novfJ, sOverflow );
	}
}

// The operation counts at zero and the substep deltas unwritten again, for
// the next launch of a step with more than FLOW_SUBSTEPS substeps.
__global__ void k_solver_refill( DWorld w, int subSteps )
{
	const float sentinel = __uint_as_float( FLOW_SENTINEL );
	for ( int b = blockIdx.x * blockDim.x + threadIdx.x; b < w.bodyCount; b += gridDim.x * blockDim.x )
	{
		w.vel[b].w = 0.0f;
		for ( int s = 0; s < subSteps; ++s )
			w.dsub[(size_t)s * w.bodyCount + b] = make_float4( sentinel, sentinel, sentinel, sentinel );
	}
}

// ---------------------------------------------------------------------------
// The solver proper: constraints as a data flow over the bodies' velocity
// rows, in one persistent launch.
//
// The reference runs its stages (per substep: warm start, solve, relax; then
// restitution) one after another, each as overflow joints, overflow contacts
// and the colours 0..10 in turn (solver.c:929-1160). All that order decides is
// in which order a body meets its constraints: two constraints without a
// common non-static body commute. So no stage is separated from the next by a
// barrier here. Every body's velocity row carries, in its fourth word, the
// number of constraint operations the body has been through in this launch; a
// constraint with the body's rank r among its d constraints runs its stage-s
// operation when that count reads s * d + r, and stores the row back with the
// count one higher. The row travels as one 16-byte relaxed access, so a row
// that shows the awaited count also shows its velocity, and no fence is
// needed. The per-substep position deltas go through rows written once per
// launch (filled with a pattern no delta has), which a reader polls the same
// way. Velocity integration is done by a body's first warm start, position
// integration by its last solve; bodies without constraints are integrated by
// a thread of their own.
//
// The bodies are dealt to the blocks in runs of their spatial order, and a
// constraint is solved in the (lower) part of its bodies. A body whose
// constraints all lie in one part lives in that block's shared memory for the
// launch; only bodies on the parts' borders go through global memory (L2).
// A warp takes up to 32 constraints of one part and colour at a time, which
// touch disjoint bodies, waits for all their bodies and runs them together.
//
// No wait is endless: every warp takes its groups in the order (stage,
// overflow joints, overflow contacts, colour), each waits only for operations
// that precede it in that order, and all blocks are resident, so the first
// unfinished group of that order is always at the head of its warp and its
// wait ends. Polls are counted all the same: a warp that makes no progress
// for flow_spin_limit polls raises the timeout bit and leaves, as do the
// others when they see the bit.
// ---------------------------------------------------------------------------
__device__ __forceinline__ float4 unpack_row( unsigned long long lo, unsigned long long hi )
{
	return make_float4( __uint_as_float( (unsigned)lo ), __uint_as_float( (unsigned)( lo >> 32 ) ),
						__uint_as_float( (unsigned)hi ), __uint_as_float( (unsigned)( hi >> 32 ) ) );
}

__device__ __forceinline__ float4 ld_row( const float4* p )
{
	unsigned long long lo, hi;
	asm volatile( "{ .reg .b128 t; ld.relaxed.gpu.global.b128 t, [%2]; mov.b128 {%0, %1}, t; }"
				  : "=l"( lo ), "=l"( hi )
				  : "l"( p )
				  : "memory" );
	return unpack_row( lo, hi );
}

__device__ __forceinline__ float4 ld_row_shared( unsigned a )
{
	unsigned long long lo, hi;
	asm volatile( "{ .reg .b128 t; ld.relaxed.cta.shared::cta.b128 t, [%2]; mov.b128 {%0, %1}, t; }"
				  : "=l"( lo ), "=l"( hi )
				  : "r"( a )
				  : "memory" );
	return unpack_row( lo, hi );
}

__device__ __forceinline__ void st_row( float4* p, float4 v )
{
	unsigned long long lo = __float_as_uint( v.x ) | ( (unsigned long long)__float_as_uint( v.y ) << 32 );
	unsigned long long hi = __float_as_uint( v.z ) | ( (unsigned long long)__float_as_uint( v.w ) << 32 );
	asm volatile( "{ .reg .b128 t; mov.b128 t, {%1, %2}; st.relaxed.gpu.global.b128 [%0], t; }" ::"l"( p ), "l"( lo ),
				  "l"( hi )
				  : "memory" );
}

__device__ __forceinline__ void st_row_shared( unsigned a, float4 v )
{
	unsigned long long lo = __float_as_uint( v.x ) | ( (unsigned long long)__float_as_uint( v.y ) << 32 );
	unsigned long long hi = __float_as_uint( v.z ) | ( (unsigned long long)__float_as_uint( v.w ) << 32 );
	asm volatile( "{ .reg .b128 t; mov.b128 t, {%1, %2}; st.relaxed.cta.shared::cta.b128 [%0], t; }" ::"r"( a ), "l"( lo ),
				  "l"( hi )
				  : "memory" );
}

// Body rows: `slot` is the body's place in this block's shared memory, or
// FLOW_NO_SLOT for a body in global memory.
#define FLOW_NO_SLOT 0xffff
struct Rows
{
	unsigned base; // shared address: velocities of all slots, then per delta row all slots
	unsigned stride; // bytes from one row kind to the next
	float4* vels;
	float4* deltas;
	float4* dsub;
	size_t cap;
	__device__ __forceinline__ float4 vel( int b, int slot ) const
	{
		return slot != FLOW_NO_SLOT ? ld_row_shared( base + 16u * (unsigned)slot ) : ld_row( vels + b );
	}
	__device__ __forceinline__ void put_vel( int b, int slot, float4 v ) const
	{
		if ( slot != FLOW_NO_SLOT )
			st_row_shared( base + 16u * (unsigned)slot, v );
		else
			st_row( vels + b, v );
	}
	// delta after s substeps of the launch
	__device__ __forceinline__ float4 delta( int s, int b, int slot ) const
	{
		if ( slot != FLOW_NO_SLOT )
			return ld_row_shared( base + stride * (unsigned)( 1 + s ) + 16u * (unsigned)slot );
		return s == 0 ? __ldcg( deltas + b ) : ld_row( dsub + ( s - 1 ) * cap + b );
	}
	__device__ __forceinline__ void put_delta( int s, bool last, int b, int slot, float4 d ) const
	{
		if ( slot != FLOW_NO_SLOT )
			st_row_shared( base + stride * (unsigned)( 1 + s ) + 16u * (unsigned)slot, d );
		else
		{
			st_row( dsub + ( s - 1 ) * cap + b, d );
			if ( last )
				__stcg( deltas + b, d );
		}
	}
};

// The two bodies of a joint or overflow contact, in registers: what their
// functions load and store. Static bodies (index < 0) read as the identity
// state and are never written (contact_solver.c:1184-1222). A joint may hold
// one body at both ends: what is stored for either end is then that body's
// state, the later store staying, as where the bodies are stored by index.
struct PairBodies
{
	int ia, ib;
	mutable BState a, b;
	__device__ __forceinline__ BState load( int i ) const
	{
		BState s;
		if ( i < 0 )
		{
			s.vx = s.vy = s.w = 0.0f;
			s.dpx = s.dpy = 0.0f;
			s.dqc = 1.0f;
			s.dqs = 0.0f;
			return s;
		}
		return i == ia ? a : b;
	}
	__device__ __forceinline__ void store( int i, const BState& s ) const
	{
		if ( i < 0 )
			return;
		if ( i == ia )
			put( a, s );
		if ( i == ib )
			put( b, s );
	}
	static __device__ __forceinline__ void put( BState& t, const BState& s )
	{
		t.vx = s.vx;
		t.vy = s.vy;
		t.w = s.w;
	}
};

// Velocity integration over a substep (solver.c:65-130) with the factors of
// k_solver_count.
__device__ __forceinline__ void integrate_velocity( const DWorld& w, const SolveParams& p, int b, BState& s )
{
	float4 r0 = w.bodyInt[2 * (size_t)b], r1 = w.bodyInt[2 * (size_t)b + 1];
	int flags = __float_as_int( r1.y );
	if ( ( flags & BI_AWAKE ) == 0 )
		return;
	fv2 v = vmuladd( mk( r0.x, r0.y ), r0.z, mk( s.vx, s.vy ) );
	float wv = r0.w + r1.x * s.w;
	float maxLinearSpeedSq = p.maxLinearSpeed * p.maxLinearSpeed;
	float maxAngularSpeedSq = p.maxAngularSpeed * p.maxAngularSpeed;
	bool capped = false;
	if ( vdot( v, v ) > maxLinearSpeedSq )
	{
		float ratio = p.maxLinearSpeed / vlen( v );
		v = vscale( ratio, v );
		capped = true;
	}
	if ( wv * wv > maxAngularSpeedSq && ( flags & BI_FAST_ROT ) == 0 )
	{
		float ratio = p.maxAngularSpeed / fabs_s( wv );
		wv *= ratio;
		capped = true;
	}
	if ( capped )
		w.bflags[b] = __ldcg( w.bflags + b ) | BF_SPEED_CAPPED;
	s.vx = v.x;
	s.vy = v.y;
	s.w = wv;
}

// Position integration over a substep (solver.c:182-200)
__device__ __forceinline__ float4 integrate_position( const DWorld& w, const SolveParams& p, int b, const BState& s )
{
	int flags = __float_as_int( w.bodyInt[2 * (size_t)b + 1].y );
	if ( ( flags & BI_AWAKE ) == 0 )
		return make_float4( s.dpx, s.dpy, s.dqc, s.dqs );
	frot dq;
	dq.c = s.dqc;
	dq.s = s.dqs;
	dq = rintegrate( dq, p.h * s.w );
	fv2 dp = vmuladd( mk( s.dpx, s.dpy ), p.h, mk( s.vx, s.vy ) );
	return make_float4( dp.x, dp.y, dq.c, dq.s );
}

// Manifold write-back of one constraint (contact_solver.c:480-509 overflow,
// :2078-2120 graph lanes; graph lanes store both points, zeros for a
// one-point manifold).
__device__ __forceinline__ void store_manifold( const DWorld& w, int c, float4 imp, float4 tot, float rolling, float rv1,
												float rv2, bool both )
{
	w.mpI[2 * c + 0] = make_float4( imp.x, imp.z, tot.x, rv1 );
	if ( both )
		w.mpI[2 * c + 1] = make_float4( imp.y, imp.w, tot.y, rv2 );
	w.mnorm[c].z = rolling;
}

// One block's work: its groups of constraints in colour order (a colour's
// joints, then its contacts) and its overflow constraints.
#define FLOW_KINDS ( 2 * F2D_OVERFLOW ) // joints of colour c at 2c, contacts at 2c + 1
#define FLOW_LIST 2048					// groups whose kind is looked up in shared memory
struct FlowPart
{
	int groupStart[FLOW_KINDS + 1]; // first group of each kind within the part
	int first[FLOW_KINDS];			// its first joint slot / group of rows
	int count[FLOW_KINDS];
	int overflow, overflowFirst; // overflow constraints and their place in ovfSorted
	unsigned char kind[FLOW_LIST];
};

// Rank of overflow constraint e on body b among the body's overflow
// constraints, from the body's (unordered) list; .y among those with
// restitution. False when the list is long: its ranks are there already.
__device__ __forceinline__ bool overflow_rank( const DWorld& w, int e, int b, int2& r )
{
	r = make_int2( 0, 0 );
	if ( b < 0 )
		return true;
	const int4 ord = w.bodyOrd[b];
	if ( ord.y > FLOW_WALK )
		return false;
	int key = ord.w - 1;
	for ( int guard = 0; key >= 0 && guard < ord.y; ++guard )
	{
		if ( ( key >> 2 ) < e )
		{
			r.x += 1;
			r.y += ( key >> 1 ) & 1;
		}
		key = w.ovfNext[2 * (size_t)( key >> 2 ) + ( key & 1 )] - 1;
	}
	return true;
}

// Ranks of overflow constraint e on both its bodies.
__device__ __forceinline__ void overflow_ranks( const DWorld& w, int e )
{
	const int novfJ = w.sc->overflowJointCount;
	int* r = (int*)( w.ovfRank + e );
	int2 bd;
	if ( e < novfJ )
		bd = w.jindex[w.overflowJoints[e]];
	else
	{
		float4 h = *krow( w, e - novfJ, KR_HEAD );
		bd = make_int2( __float_as_int( h.x ), __float_as_int( h.y ) );
	}
	for ( int side = 0; side < 2; ++side )
	{
		int2 k;
		if ( overflow_rank( w, e, side ? bd.y : bd.x, k ) )
		{
			r[side] = k.x;
			r[2 + side] = k.y;
		}
	}
}

// Lanes of a block for `n` overflow constraints: a quarter of the warps at
// most, whose chains would hold up the colour groups of a warp that had both.
__device__ __forceinline__ int overflow_lanes( int threads, int n )
{
	return 32 * min( threads / 128, n );
}

__device__ __forceinline__ void flow_part( const DWorld& w, const SolveParams& p, int part, FlowPart& f )
{
	const int novf = w.sc->overflowCount + w.sc->overflowJointCount;
	if ( threadIdx.x < FLOW_KINDS )
	{
		int k = threadIdx.x, bin = part * F2D_OVERFLOW + ( k >> 1 );
		bool contacts = k & 1;
		f.first[k] = contacts ? w.binContactStart[bin] : ( w.jointCount > 0 ? w.binJointStart[bin] : 0 );
		f.count[k] = contacts ? w.binContacts[bin] : ( w.jointCount > 0 ? w.binJoints[bin] : 0 );
	}
	if ( threadIdx.x == FLOW_KINDS )
	{
		f.overflow = novf > 0 ? w.binOverflow[part] : 0;
		f.overflowFirst = novf > 0 ? w.binOverflowStart[part] : 0;
	}
	__syncthreads();
	if ( threadIdx.x == 0 )
	{
		int at = 0;
		for ( int k = 0; k < FLOW_KINDS; ++k )
		{
			f.groupStart[k] = at;
			at += ( f.count[k] + 31 ) >> 5;
		}
		f.groupStart[FLOW_KINDS] = at;
	}
	// overflow constraints in their serial order: each counts the smaller ones
	if ( f.overflow <= FLOW_SORT )
		for ( int i = threadIdx.x; i < f.overflow; i += blockDim.x )
		{
			int e = w.ovfItems[f.overflowFirst + i], rank = 0;
			for ( int j = 0; j < f.overflow; ++j )
				rank += w.ovfItems[f.overflowFirst + j] < e ? 1 : 0;
			w.ovfSorted[f.overflowFirst + rank] = e;
		}
	// more than a lane each: their ranks before any of them starts, as a walk
	// between two operations would hold up the lanes beside it
	if ( f.overflow > overflow_lanes( blockDim.x, f.overflow ) )
		for ( int i = threadIdx.x; i < f.overflow; i += blockDim.x )
			overflow_ranks( w, w.ovfItems[f.overflowFirst + i] );
	__syncthreads();
	for ( int g = threadIdx.x; g < min( f.groupStart[FLOW_KINDS], FLOW_LIST ); g += blockDim.x )
	{
		int k = 0;
		while ( k < FLOW_KINDS - 1 && g >= f.groupStart[k + 1] )
			k += 1;
		f.kind[g] = (unsigned char)k;
	}
	__syncthreads();
}

// A constraint's view of one body: KR_REF packs the bodies (x, y), their
// slots (z, 16 bits each) and per body, 9 bits from bit 0 and bit 16 of w: the
// colour's rank among the body's colours, their number, and whether overflow
// constraints lead them.
__device__ __forceinline__ int ref_bits( const int4& ord, int colour )
{
	unsigned bits = (unsigned)ord.x & FLOW_COLOURS;
	return __popc( bits & ( ( 1u << colour ) - 1u ) ) | ( __popc( bits ) << 4 ) | ( ord.y > 0 ? 256 : 0 );
}

// A body has a slot when its constraints all lie in this part and its place
// fits the shared memory.
__device__ __forceinline__ int body_slot( const DWorld& w, const int4& ord, int b, int firstPos, int slots )
{
	int pos = w.bodyPos[b];
	if ( pos < 0 || ( ord.x & FLOW_GLOBAL ) || pos - firstPos >= slots )
		return FLOW_NO_SLOT;
	return pos - firstPos;
}

// Loads the rows of a contact constraint (all of them, or those its warm
// start needs).
__device__ __forceinline__ void load_lane( const float4* row, Lane& L, bool all )
{
	L.ms = row[32 * KR_MASS];
	L.nm = row[32 * KR_NORMAL];
	L.misc = row[32 * KR_MISC];
	L.imp = row[32 * KR_IMP];
	L.an[0] = row[32 * KR_ANCH1];
	L.an[1] = row[32 * KR_ANCH2];
	if ( all )
	{
		L.pt[0] = row[32 * KR_P1];
		L.pt[1] = row[32 * KR_P2];
		L.tot = row[32 * KR_TOT];
	}
}

__device__ __forceinline__ void store_lane( float4* row, const Lane& L )
{
	row[32 * KR_IMP] = L.imp;
	row[32 * KR_TOT] = L.tot;
	row[32 * KR_MISC] = L.misc;
}

// One constraint's pair of bodies and where their rows are.
struct FlowPair
{
	int ia, ib;		  // -1 static
	int slotA, slotB; // FLOW_NO_SLOT: global
	int rankA, rankB, degA, degB;
};

// What a waiting constraint has seen of its bodies.
struct FlowSeen
{
	float4 vA, vB, dA, dB;
	bool okA, okB, okD;
};

// One poll of the rows a constraint still waits for; true when it has all.
// `ds`: substep delta rows, -1 when the operation needs none.
__device__ __forceinline__ bool flow_poll( const Rows& rows, const FlowPair& q, int wantA, int wantB, int ds, FlowSeen& s )
{
	float4 a, b;
	if ( !s.okA )
		a = rows.vel( q.ia, q.slotA );
	if ( !s.okB )
		b = rows.vel( q.ib, q.slotB );
	if ( !s.okD && ds >= 0 )
	{
		s.dA = s.dB = make_float4( 0.0f, 0.0f, 1.0f, 0.0f );
		if ( q.ia >= 0 )
			s.dA = rows.delta( ds, q.ia, q.slotA );
		if ( q.ib >= 0 )
			s.dB = rows.delta( ds, q.ib, q.slotB );
		s.okD = __float_as_uint( s.dA.x ) != FLOW_SENTINEL && __float_as_uint( s.dB.x ) != FLOW_SENTINEL;
	}
	if ( !s.okA )
	{
		s.vA = a;
		s.okA = __float_as_int( a.w ) == wantA;
	}
	if ( !s.okB )
	{
		s.vB = b;
		s.okB = __float_as_int( b.w ) == wantB;
	}
	return s.okA && s.okB && ( s.okD || ds < 0 );
}

__device__ __forceinline__ void flow_expect( const FlowPair& q, FlowSeen& s )
{
	s.okA = q.ia < 0;
	s.okB = q.ib < 0;
	if ( s.okA )
		s.vA = make_float4( 0.0f, 0.0f, 0.0f, 0.0f );
	if ( s.okB )
		s.vB = make_float4( 0.0f, 0.0f, 0.0f, 0.0f );
}

__device__ __forceinline__ void flow_states( const FlowPair& q, const FlowSeen& s, PairBodies& ba )
{
	ba.ia = q.ia;
	ba.ib = q.ib;
	ba.a = { s.vA.x, s.vA.y, s.vA.z, s.dA.x, s.dA.y, s.dA.z, s.dA.w };
	ba.b = { s.vB.x, s.vB.y, s.vB.z, s.dB.x, s.dB.y, s.dB.z, s.dB.w };
}

// The velocity rows back with their counts one higher; after a body's last
// solve of a substep, its new delta. One body at both ends has one row, written
// once: the body's next constraint may have passed on from it by a second
// write.
__device__ __forceinline__ void flow_publish( const DWorld& w, const SolveParams& p, const Rows& rows, const FlowPair& q,
											  const PairBodies& ba, int wantA, int wantB, int sub, bool solve )
{
	const bool one = q.ia == q.ib;
	if ( q.ia >= 0 && !one )
		rows.put_vel( q.ia, q.slotA, make_float4( ba.a.vx, ba.a.vy, ba.a.w, __int_as_float( wantA + 1 ) ) );
	if ( q.ib >= 0 )
		rows.put_vel( q.ib, q.slotB, make_float4( ba.b.vx, ba.b.vy, ba.b.w, __int_as_float( wantB + 1 ) ) );
	if ( solve )
	{
		const bool last = sub == p.subSteps - 1;
		if ( q.ia >= 0 && !one && q.rankA == q.degA - 1 )
			rows.put_delta( sub + 1, last, q.ia, q.slotA, integrate_position( w, p, q.ia, ba.a ) );
		if ( q.ib >= 0 && q.rankB == q.degB - 1 )
			rows.put_delta( sub + 1, last, q.ib, q.slotB, integrate_position( w, p, q.ib, ba.b ) );
	}
}

__device__ __forceinline__ int flow_spin_limit( const DWorld& w )
{
	return FLOW_SPIN_LIMIT + FLOW_SPIN_OVERFLOW * min( w.sc->overflowCount + w.sc->overflowJointCount, FLOW_OVERFLOW_MOST );
}

// Counts a poll without progress; true when the wait is to be given up.
__device__ __forceinline__ bool flow_give_up( const DWorld& w, int& spins )
{
	spins += 1;
	if ( ( spins & 1023 ) != 0 )
		return false;
	bool out = spins >= flow_spin_limit( w );
	if ( out && ( threadIdx.x & 31 ) == 0 )
		atomicOr( &w.sc->error, F2D_ERR_BARRIER_TIMEOUT );
	return __any_sync( 0xffffffffu, out || ( ld_relaxed_s32( &w.sc->error ) & F2D_ERR_BARRIER_TIMEOUT ) );
}

// One warp's groups first, first + stride, ... of the part's colours, through
// every stage.
__device__ __forceinline__ void solve_colours( const DWorld& w, const SolveParams& p, const Rows& rows, const FlowPart& f,
											   int firstPos, int slots, int first, int stride )
{
	const int lane = threadIdx.x & 31;
	const int nGroups = f.groupStart[FLOW_KINDS];
	const int stages = 3 * p.subSteps; // restitution is stage `stages`
	const int lastStage = p.restitution ? stages : stages - 1;
	if ( first >= nGroups )
		return;
	const bool single = first + stride >= nGroups; // the group stays in registers

	Lane L;
	float4* row = nullptr;
	int joint = -1; // joint of this lane, -1 in a group of contacts
	bool item = false;
	FlowPair q = { -1, -1, FLOW_NO_SLOT, FLOW_NO_SLOT, 0, 0, 1, 1 };
	FlowSeen s;
	s.dA = s.dB = make_float4( 0.0f, 0.0f, 1.0f, 0.0f );
	s.okD = false;

	for ( int stage = 0; stage <= lastStage; ++stage )
	{
		const int sub = stage / 3;
		const bool rest = stage == stages;
		const int op = rest ? 3 : stage - 3 * sub; // 0 warm start, 1 solve, 2 relax, 3 restitution
		for ( int g = first; g < nGroups; g += stride )
		{
			if ( !single || stage == 0 || rest )
			{
				// open the group
				int k = 0;
				if ( g < FLOW_LIST )
					k = f.kind[g];
				else
					while ( k < FLOW_KINDS - 1 && g >= f.groupStart[k + 1] )
						k += 1;
				const int gk = g - f.groupStart[k];
				item = 32 * gk + lane < f.count[k];
				joint = -1;
				if ( k & 1 )
				{
					row = w.kRow + (size_t)( f.first[k] + gk ) * ( KROWS * 32 ) + lane;
					load_lane( row, L, op != 0 || single );
				}
				else
					joint = w.jointSlots[f.first[k] + ( item ? 32 * gk + lane : 0 )];
				if ( joint < 0 && stage > 0 && !rest )
				{
					float4 r = row[32 * KR_REF];
					q.ia = __float_as_int( r.x );
					q.ib = __float_as_int( r.y );
					q.slotA = __float_as_int( r.z ) & 0xffff;
					q.slotB = (unsigned)__float_as_int( r.z ) >> 16;
					int bits = __float_as_int( r.w );
					q.rankA = bits & 15;
					q.degA = ( bits >> 4 ) & 15;
					q.rankB = ( bits >> 16 ) & 15;
					q.degB = ( bits >> 20 ) & 15;
					if ( item && ( bits & 256 ) )
					{
						int lead = w.bodyOrd[q.ia].y;
						q.rankA += lead;
						q.degA += lead;
					}
					if ( item && ( bits & ( 256 << 16 ) ) )
					{
						int lead = w.bodyOrd[q.ib].y;
						q.rankB += lead;
						q.degB += lead;
					}
				}
				else if ( item )
				{
					if ( joint < 0 )
					{
						float4 h = row[32 * KR_HEAD];
						q.ia = __float_as_int( h.x );
						q.ib = __float_as_int( h.y );
					}
					else
					{
						int2 idx = w.jindex[joint];
						q.ia = idx.x;
						q.ib = idx.y;
					}
					const int colour = k >> 1;
					int4 oa = make_int4( 0, 0, 0, 0 ), ob = oa;
					if ( q.ia >= 0 )
						oa = w.bodyOrd[q.ia];
					if ( q.ib >= 0 )
						ob = w.bodyOrd[q.ib];
					q.slotA = q.ia >= 0 ? body_slot( w, oa, q.ia, firstPos, slots ) : FLOW_NO_SLOT;
					q.slotB = q.ib >= 0 ? body_slot( w, ob, q.ib, firstPos, slots ) : FLOW_NO_SLOT;
					q.degA = oa.y + __popc( oa.x & FLOW_COLOURS );
					q.degB = ob.y + __popc( ob.x & FLOW_COLOURS );
					unsigned below = ( 1u << colour ) - 1u;
					int shift = rest ? FLOW_REST_SHIFT : 0;
					q.rankA = ( rest ? oa.z : oa.y ) + __popc( ( (unsigned)oa.x >> shift ) & below );
					q.rankB = ( rest ? ob.z : ob.y ) + __popc( ( (unsigned)ob.x >> shift ) & below );
					if ( joint < 0 && !single && stage == 0 )
						row[32 * KR_REF] = make_float4(
							__int_as_float( q.ia ), __int_as_float( q.ib ), __int_as_float( q.slotA | ( q.slotB << 16 ) ),
							__int_as_float( ref_bits( oa, colour ) | ( ref_bits( ob, colour ) << 16 ) ) );
				}
				if ( rest )
					item = item && joint < 0 && L.misc.x != 0.0f; // contacts that have some
				if ( !item )
					q.ia = q.ib = -1;
				s.okD = false;
			}
			else if ( op == 2 )
				s.okD = false; // relaxing reads the substep's new deltas

			// wait for the operations before this one on every body of the group
			// (the restitution counts follow the last relax stage's)
			const int wantA = stage * q.degA + q.rankA, wantB = stage * q.degB + q.rankB;
			// deltas: none for restitution and a contact's warm start
			const int ds = rest || ( op == 0 && joint < 0 ) ? -1 : sub + ( op == 2 ? 1 : 0 );
			flow_expect( q, s );
			for ( int spins = 0; !__all_sync( 0xffffffffu, flow_poll( rows, q, wantA, wantB, ds, s ) ); )
				if ( flow_give_up( w, spins ) )
					return;

			if ( item )
			{
				PairBodies ba;
				flow_states( q, s, ba );
				if ( op == 0 )
				{
					if ( q.ia >= 0 && q.rankA == 0 )
						integrate_velocity( w, p, q.ia, ba.a );
					if ( q.ib >= 0 && q.rankB == 0 )
						integrate_velocity( w, p, q.ib, ba.b );
				}
				if ( joint < 0 )
				{
					Soft soft = ( q.ia < 0 || q.ib < 0 ) ? p.staticSoft : p.contactSoft;
					if ( op == 0 )
						lane_warm( ba.a, ba.b, L );
					else if ( op == 3 )
						lane_restitution( ba.a, ba.b, L, p.restitutionThreshold );
					else
						lane_solve( ba.a, ba.b, L, soft, p.inv_h, p.minBiasVel, op == 1 );
				}
				else if ( op == 0 )
					joint_warm_start( w, ba, joint );
				else
					joint_solve( w, ba, joint, p.h, p.inv_h, op == 1 );
				flow_publish( w, p, rows, q, ba, wantA, wantB, sub, op == 1 );
				// the step's last operation of a contact hands its impulses over
				if ( joint < 0 )
				{
					if ( p.restitution && ( rest || ( stage == stages - 1 && L.misc.x == 0.0f ) ) )
						store_manifold( w, __float_as_int( row[32 * KR_HEAD].z ), L.imp, L.tot, L.misc.w, L.pt[0].w, L.pt[1].w,
										true );
					else if ( op != 0 && ( !single || stage == stages - 1 ) )
						store_lane( row, L );
				}
			}
			__syncwarp();
		}
	}
}

// Overflow constraints: each lane goes through its own, first, first +
// stride, ... of the part's list, at its own pace; a round polls for all
// lanes and runs those that are ready.
__device__ __forceinline__ void solve_overflows( const DWorld& w, const SolveParams& p, const Rows& rows,
												 const FlowPart& f, int firstPos, int slots, int first, int stride )
{
	const int stages = 3 * p.subSteps;
	const int novfJ = w.sc->overflowJointCount;
	const bool single = first + stride >= f.overflow;
	Lane L;
	float4* row = nullptr;
	int joint = -1, contact = -1, points = 0;
	FlowPair q = { -1, -1, FLOW_NO_SLOT, FLOW_NO_SLOT, 0, 0, 1, 1 };
	FlowSeen s;
	s.dA = s.dB = make_float4( 0.0f, 0.0f, 1.0f, 0.0f );
	int i = first, stage = 0;
	bool act = i < f.overflow, fresh = true;
	if ( act && f.overflow <= stride )
		overflow_ranks( w, w.ovfSorted[f.overflowFirst + i] );
	for ( int spins = 0;; )
	{
		const bool rest = stage == stages;
		const int sub = stage / 3;
		const int op = rest ? 3 : stage - 3 * sub;
		bool fire = false;
		if ( act )
		{
			if ( fresh )
			{
				int e = w.ovfSorted[f.overflowFirst + i];
				joint = e < novfJ ? w.overflowJoints[e] : -1;
				if ( joint >= 0 )
				{
					int2 idx = w.jindex[joint];
					q.ia = idx.x;
					q.ib = idx.y;
				}
				else
				{
					row = krow( w, e - novfJ, 0 );
					load_lane( row, L, true );
					float4 h = row[32 * KR_HEAD];
					q.ia = __float_as_int( h.x );
					q.ib = __float_as_int( h.y );
					contact = __float_as_int( h.z );
					points = __float_as_int( h.w );
				}
				int4 oa = make_int4( 0, 0, 0, 0 ), ob = oa;
				if ( q.ia >= 0 )
					oa = w.bodyOrd[q.ia];
				if ( q.ib >= 0 )
					ob = w.bodyOrd[q.ib];
				q.slotA = q.ia >= 0 ? body_slot( w, oa, q.ia, firstPos, slots ) : FLOW_NO_SLOT;
				q.slotB = q.ib >= 0 ? body_slot( w, ob, q.ib, firstPos, slots ) : FLOW_NO_SLOT;
				q.degA = oa.y + __popc( oa.x & FLOW_COLOURS );
				q.degB = ob.y + __popc( ob.x & FLOW_COLOURS );
				int4 o = w.ovfRank[e];
				q.rankA = rest ? o.z : o.x;
				q.rankB = rest ? o.w : o.y;
				fresh = false;
				s.okD = false;
				flow_expect( q, s );
			}
			const int wantA = stage * q.degA + q.rankA, wantB = stage * q.degB + q.rankB;
			const int ds = rest || ( op == 0 && joint < 0 ) ? -1 : sub + ( op == 2 ? 1 : 0 );
			fire = flow_poll( rows, q, wantA, wantB, ds, s );
			if ( fire )
			{
				PairBodies ba;
				flow_states( q, s, ba );
				if ( op == 0 )
				{
					if ( q.ia >= 0 && q.rankA == 0 )
						integrate_velocity( w, p, q.ia, ba.a );
					if ( q.ib >= 0 && q.rankB == 0 )
						integrate_velocity( w, p, q.ib, ba.b );
				}
				if ( joint < 0 )
				{
					Soft soft = ( q.ia < 0 || q.ib < 0 ) ? p.staticSoft : p.contactSoft;
					if ( op == 0 )
						warm_overflow( ba.a, ba.b, L, points );
					else if ( op == 3 )
						restitution_overflow( ba.a, ba.b, L, points, p.restitutionThreshold );
					else
						solve_overflow( ba.a, ba.b, L, points, soft, p.inv_h, p.pushout, op == 1 );
				}
				else if ( op == 0 )
					joint_warm_start( w, ba, joint );
				else
					joint_solve( w, ba, joint, p.h, p.inv_h, op == 1 );
				flow_publish( w, p, rows, q, ba, wantA, wantB, sub, op == 1 );
				if ( joint < 0 )
				{
					if ( p.restitution && ( rest || ( stage == stages - 1 && L.misc.x == 0.0f ) ) )
						store_manifold( w, contact, L.imp, L.tot, L.misc.w, L.pt[0].w, L.pt[1].w, points > 1 );
					else if ( op != 0 && ( !single || stage == stages - 1 ) )
						store_lane( row, L );
				}
				// this lane's next operation
				if ( !single )
				{
					fresh = true;
					i += stride;
					if ( i >= f.overflow )
					{
						i = first;
						stage += 1;
					}
				}
				else
				{
					stage += 1;
					if ( stage % 3 == 2 )
						s.okD = false; // relaxing reads the substep's new deltas
					flow_expect( q, s );
				}
				if ( stage >= stages )
				{
					// restitution: contacts that have some
					fresh = true;
					act = false;
					while ( stage == stages && p.restitution && i < f.overflow )
					{
						int e = w.ovfSorted[f.overflowFirst + i];
						if ( e >= novfJ && krow( w, e - novfJ, KR_MISC )->x != 0.0f )
						{
							act = true;
							break;
						}
						i += stride;
					}
				}
			}
		}
		if ( !__any_sync( 0xffffffffu, act ) )
			return;
		if ( __any_sync( 0xffffffffu, fire ) )
			spins = 0;
		else if ( flow_give_up( w, spins ) )
			return;
	}
}

template <int THREADS>
__global__ void __launch_bounds__( THREADS ) k_solve( DWorld w, SolveParams p )
{
	extern __shared__ float4 sbody[]; // velocities of all slots, deltas at the start, deltas after each substep
	__shared__ FlowPart f;
	const int part = blockIdx.x;
	const int chunk = part_chunk( w, p );
	const int firstPos = part * chunk;
	const int mine = max( min( min( w.sc->orderTotal - firstPos, chunk ), p.slots ), 0 );
	const float sentinel = __uint_as_float( FLOW_SENTINEL );
	for ( int t = threadIdx.x; t < mine; t += THREADS )
	{
		int b = w.bodyAt[firstPos + t];
		float4 v = __ldcg( w.vel + b );
		v.w = 0.0f;
		sbody[t] = v;
		sbody[p.slots + t] = __ldcg( w.delta + b );
		for ( int k = 0; k < p.subSteps; ++k )
			sbody[( 2 + k ) * p.slots + t] = make_float4( sentinel, sentinel, sentinel, sentinel );
	}
	flow_part( w, p, part, f );
	// bodies no constraint holds: all substeps at once, nothing to wait for
	// (the last blocks first: a small world's parts are the first ones)
	for ( int b = ( gridDim.x - 1 - blockIdx.x ) * THREADS + threadIdx.x; b < w.bodyCount; b += gridDim.x * THREADS )
	{
		int4 o = w.bodyOrd[b];
		if ( ( o.x & FLOW_COLOURS ) != 0 || o.y != 0 ||
			 ( __float_as_int( w.bodyInt[2 * (size_t)b + 1].y ) & BI_AWAKE ) == 0 )
			continue;
		float4 v = w.vel[b], d = w.delta[b];
		BState s = { v.x, v.y, v.z, d.x, d.y, d.z, d.w };
		for ( int sub = 0; sub < p.subSteps; ++sub )
		{
			integrate_velocity( w, p, b, s );
			d = integrate_position( w, p, b, s );
			s.dpx = d.x;
			s.dpy = d.y;
			s.dqc = d.z;
			s.dqs = d.w;
		}
		w.vel[b] = make_float4( s.vx, s.vy, s.w, 0.0f );
		w.delta[b] = d;
	}
	const Rows rows = { (unsigned)__cvta_generic_to_shared( sbody ), 16u * (unsigned)p.slots, w.vel, w.delta, w.dsub,
						(size_t)w.bodyCount };
	const int warp = threadIdx.x >> 5, warps = THREADS / 32;
	const int ovfWarps = overflow_lanes( THREADS, f.overflow ) / 32;
	if ( warp < warps - ovfWarps )
		solve_colours( w, p, rows, f, firstPos, mine, warp, warps - ovfWarps );
	else
		solve_overflows( w, p, rows, f, firstPos, mine, ( threadIdx.x & 31 ) * ovfWarps + warp - ( warps - ovfWarps ),
						 32 * ovfWarps );
	__syncthreads();
	for ( int t = threadIdx.x; t < mine; t += THREADS )
	{
		int b = w.bodyAt[firstPos + t];
		int4 o = w.bodyOrd[b];
		if ( ( o.x & FLOW_GLOBAL ) || ( ( o.x & FLOW_COLOURS ) == 0 && o.y == 0 ) )
			continue;
		float4 v = sbody[t];
		w.vel[b] = make_float4( v.x, v.y, v.z, 0.0f );
		w.delta[b] = sbody[( 1 + p.subSteps ) * p.slots + t];
	}
}

// A launch of nothing but grid barriers on one block per SM: what a barrier
// per stage would cost at least.
__global__ void __launch_bounds__( 512 ) k_barrier_probe( unsigned* counter, int* err, int n )
{
	unsigned epoch = 0;
	for ( int i = 0; i < n; ++i )
		if ( !grid_barrier( counter, err, epoch ) )
			return;
}

float solver_barrier_probe( StepScratch& s, cudaStream_t st, unsigned* counter, int* err, int n )
{
	cudaEvent_t a, b;
	cudaEventCreate( &a );
	cudaEventCreate( &b );
	cudaMemsetAsync( counter, 0, sizeof( unsigned ), st );
	void* args[] = { &counter, &err, &n };
	cudaEventRecord( a, st );
	cudaLaunchCooperativeKernel( (void*)k_barrier_probe, dim3( s.solverBlocks ), dim3( 512 ), args, 0, st );
	cudaEventRecord( b, st );
	cudaEventSynchronize( b );
	float ms = 0.0f;
	cudaEventElapsedTime( &ms, a, b );
	cudaEventDestroy( a );
	cudaEventDestroy( b );
	return n > 0 ? 1000.0f * ms / (float)n : 0.0f;
}

// ---------------------------------------------------------------------------
// host driver
// ---------------------------------------------------------------------------
#define SOLVER_ROWS_SMEM ( 120 * 1024 ) // body rows a block keeps, at most; the rest caches constraint rows
// Threads per SM: twelve warps. Measured (100k pile at its densest, 25k pile,
// 820-box pyramid; us per launch): 256 threads 425, 187, 129; 320: 327, 172,
// 121; 384: 312, 172, 119; 512: 335, 198, 133; 768: 467, 257, 150. More warps
// cost registers (spills from 512 on) and issue slots (waiting warps poll);
// fewer leave too many groups to a warp.
#define SOLVER_THREADS 384

static size_t solver_smem( int slots, int subSteps )
{
	return 16u * (size_t)( 2 + subSteps ) * slots;
}

// Co-resident grid of `perSM` blocks per SM.
template <int THREADS> static int grid_blocks( int perSM )
{
	int fit = 0, dev = 0, sms = 0;
	size_t smem = SOLVER_ROWS_SMEM / perSM;
	if ( cudaFuncSetAttribute( k_solve<THREADS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem ) != cudaSuccess )
		return 0;
	cudaOccupancyMaxActiveBlocksPerMultiprocessor( &fit, k_solve<THREADS>, THREADS, smem );
	cudaGetDevice( &dev );
	cudaDeviceGetAttribute( &sms, cudaDevAttrMultiProcessorCount, dev );
	int blocks = sms * ( fit < perSM ? fit : perSM );
	return blocks < SOLVER_MAX_PARTS ? blocks : SOLVER_MAX_PARTS;
}

int solver_max_blocks( int perSM )
{
	return perSM == 2 ? grid_blocks<SOLVER_THREADS / 2>( 2 ) : grid_blocks<SOLVER_THREADS>( 1 );
}

// The bodies' spatial order and cleared tables, on a stream of their own
// beside the collide phase: they need the leaf order and the last step's
// colours only.
// What the body order and the set-up after it start from, in one launch (five
// memset nodes of some 1.5 us each before).
__global__ void k_order_clear( DWorld w, int tiles, int subSteps )
{
	const int tid = blockIdx.x * blockDim.x + threadIdx.x, stride = gridDim.x * blockDim.x;
	for ( int i = tid; i < tiles + 2; i += stride )
		w.orderState[i] = 0ull;
	for ( int i = tid; i < SOLVER_MAX_PARTS * ( 2 * F2D_OVERFLOW + 1 ) + 1; i += stride )
		w.binContacts[i] = 0; // and flowLong
	for ( int i = tid; i < w.bodyCount; i += stride )
	{
		w.bodyPos[i] = -1;
		w.bodyOrd[i] = make_int4( 0, 0, 0, 0 );
	}
	const float ones = __int_as_float( -1 );
	for ( size_t i = tid; i < (size_t)w.bodyCount * subSteps; i += stride )
		w.dsub[i] = make_float4( ones, ones, ones, ones );
}

void launch_solver_order( DWorld& w, StepScratch& s, cudaStream_t st )
{
	int tiles = ( w.shapeCap + ORDER_TILE - 1 ) / ORDER_TILE;
	int subSteps = s.subSteps < FLOW_SUBSTEPS ? s.subSteps : FLOW_SUBSTEPS;
	k_order_clear<<<grid_for( w.bodyCount ), 256, 0, st>>>( w, tiles, subSteps );
	k_body_order<<<tiles, ORDER_THREADS, 0, st>>>( w );
}

void launch_solver( DWorld& w, StepScratch& s, cudaStream_t st, float dt, int subSteps )
{
	SolveParams p;
	p.dt = dt;
	p.inv_dt = 1.0f / dt;
	p.h = dt / (float)subSteps;
	p.inv_h = (float)subSteps * p.inv_dt;
	float contactHertz = fmin_s( w.contactHertz, 0.125f * p.inv_h );
	p.contactSoft = make_soft( contactHertz, w.contactDampingRatio, p.h );
	p.staticSoft = make_soft( 2.0f * contactHertz, w.contactDampingRatio, p.h );
	float contactSpeed = w.maxContactPushSpeed / p.staticSoft.massScale;
	p.minBiasVel = -contactSpeed;
	p.pushout = w.maxContactPushSpeed;
	float jointHertz = fmin_s( w.jointHertz, 0.25f * p.inv_h );
	p.jointSoft = make_soft( jointHertz, w.jointDampingRatio, p.h );
	p.restitutionThreshold = w.restitutionThreshold;
	p.maxLinearSpeed = w.maxLinearSpeed;
	p.maxAngularSpeed = F2D_MAX_ROTATION * p.inv_dt;
	p.gravity = w.gravity;
	p.enableWarmStarting = w.enableWarmStarting;
	p.subSteps = subSteps < FLOW_SUBSTEPS ? subSteps : FLOW_SUBSTEPS;

	const bool two = s.solverVariant == SOLVER_TWO_PER_SM && s.solverBlocks2 > 0;
	p.parts = two ? s.solverBlocks2 : s.solverBlocks;
	p.minChunk = s.smallParts ? SOLVER_SMALL_CHUNK : SOLVER_MIN_CHUNK;
	p.onePart = s.smallParts ? 0 : ( s.solverVariant == SOLVER_FEW_PARTS ? SOLVER_FEW_MOST * SOLVER_ONE_PART : SOLVER_ONE_PART );
	int fit = ( two ? SOLVER_ROWS_SMEM / 2 : SOLVER_ROWS_SMEM ) / ( 16 * ( 2 + p.subSteps ) );
	int want = ( w.bodyCount + p.parts - 1 ) / p.parts;
	want = want > p.minChunk ? want : p.minChunk;
	want = want > p.onePart ? want : p.onePart;
	want = want < w.bodyCount ? want : w.bodyCount;
	p.slots = want < fit ? want : fit;

	k_solver_count<<<grid_for( w.contactCap ), 256, 0, st>>>( w, p );
	size_t binSmem = sizeof( int ) * (size_t)p.parts * ( 2 * F2D_OVERFLOW + 1 );
	k_solver_prepare<<<grid_for( w.contactCap ), 256, binSmem, st>>>( w, p );
	if ( w.jointCount > 0 )
		launch_prepare_joints( w, st, p.h, p.jointSoft );
	if ( w.learnMode & 2 )
		launch_learned_warm_start( w, st );
	if ( s.evSolveStart )
		cudaEventRecord( s.evSolveStart, st );
	for ( int done = 0; done < subSteps; done += p.subSteps )
	{
		p.subSteps = subSteps - done < FLOW_SUBSTEPS ? subSteps - done : FLOW_SUBSTEPS;
		p.restitution = done + p.subSteps == subSteps;
		if ( done > 0 )
			k_solver_refill<<<grid_for( w.bodyCount ), 256, 0, st>>>( w, p.subSteps );
		void* args[] = { &w, &p };
		size_t smem = solver_smem( p.slots, p.subSteps );
		if ( two )
			cudaLaunchCooperativeKernel( (void*)k_solve<SOLVER_THREADS / 2>, dim3( p.parts ), dim3( SOLVER_THREADS / 2 ), args,
										 smem, st );
		else
			cudaLaunchCooperativeKernel( (void*)k_solve<SOLVER_THREADS>, dim3( p.parts ), dim3( SOLVER_THREADS ), args, smem, st );
	}
}
