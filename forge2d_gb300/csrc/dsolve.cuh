// Constraint arithmetic of the soft-step solver.
//
// Graph-colour contacts follow the operand order of the reference's SIMD
// lanes (packages/forge2d/third_party/box2d/src/contact_solver.c:1438-2120,
// separate mul and add, SSE2 min/max/blend semantics); overflow contacts
// follow its scalar functions (contact_solver.c:24-510). Built with
// -fmad=false the results are bit-identical to the reference C code.
#pragma once

#include "dworld.cuh"

// Rows of a contact constraint: slot k's row r is lane k % 32 of row r of
// block k / 32, so the 32 constraints of a group read each row in one
// coalesced access at a constant offset from one address.
#define KR_HEAD 0	// body A, body B (-1 static), contact, point count
#define KR_REF 1	// the solver's view of the bodies (solver.cu)
#define KR_MASS 2	// invMassA invIA invMassB invIB
#define KR_NORMAL 3 // normal.x normal.y friction tangentSpeed
#define KR_MISC 4	// restitution rollingResistance rollingMass rollingImpulse
#define KR_IMP 5	// normalImpulse1 normalImpulse2 tangentImpulse1 tangentImpulse2
#define KR_ANCH1 6	// anchorA1.xy anchorB1.xy
#define KR_ANCH2 7	// anchorA2.xy anchorB2.xy
#define KR_P1 8		// baseSeparation normalMass tangentMass relativeVelocity (point 1)
#define KR_P2 9		// same, point 2
#define KR_TOT 10	// totalNormalImpulse1 totalNormalImpulse2

__device__ __forceinline__ float4* krow( const DWorld& w, int k, int row )
{
	return w.kRow + ( (size_t)( k >> 5 ) * KROWS + row ) * 32 + ( k & 31 );
}

__device__ __forceinline__ float lmax( float a, float b )
{
	return a > b ? a : b;
}
__device__ __forceinline__ float lmin( float a, float b )
{
	return a < b ? a : b;
}

// A contact constraint of a colour in registers.
struct Lane
{
	float4 ms;	 // KR_MASS
	float4 nm;	 // KR_NORMAL
	float4 misc; // KR_MISC
	float4 imp;	 // KR_IMP
	float4 tot;	 // KR_TOT
	float4 an[2];
	float4 pt[2];
};

// contact_solver.c:1671-1727
__device__ __forceinline__ void lane_warm( BState& A, BState& B, const Lane& L )
{
	const float4 ms = L.ms, nm = L.nm;
	float tx = nm.y;
	float ty = 0.0f - nm.x;
	float nis[2] = { L.imp.x, L.imp.y };
	float tis[2] = { L.imp.z, L.imp.w };
	for ( int j = 0; j < 2; ++j )
	{
		float rAx = L.an[j].x, rAy = L.an[j].y, rBx = L.an[j].z, rBy = L.an[j].w;
		float Px = nis[j] * nm.x + tis[j] * tx;
		float Py = nis[j] * nm.y + tis[j] * ty;
		A.w = A.w - ms.y * ( rAx * Py - rAy * Px );
		A.vx = A.vx - ms.x * Px;
		A.vy = A.vy - ms.x * Py;
		B.w = B.w + ms.w * ( rBx * Py - rBy * Px );
		B.vx = B.vx + ms.z * Px;
		B.vy = B.vy + ms.z * Py;
	}
	A.w = A.w - ms.y * L.misc.w;
	B.w = B.w + ms.w * L.misc.w;
}

// contact_solver.c:1729-1967
__device__ __forceinline__ void lane_solve( BState& A, BState& B, Lane& L, Soft soft, float inv_h, float minBiasVel,
											bool useBias )
{
	const float4 ms = L.ms, nm = L.nm;
	float4 misc = L.misc;
	float biasRate, massScale, impulseScale;
	if ( useBias )
	{
		biasRate = soft.biasRate;
		massScale = soft.massScale;
		impulseScale = soft.impulseScale;
	}
	else
	{
		biasRate = 0.0f;
		massScale = 1.0f;
		impulseScale = 0.0f;
	}
	float totalNormalImpulse = 0.0f;
	float dpx = B.dpx - A.dpx;
	float dpy = B.dpy - A.dpy;
	float nis[2] = { L.imp.x, L.imp.y };
	float tis[2] = { L.imp.z, L.imp.w };
	float tots[2] = { L.tot.x, L.tot.y };
	for ( int j = 0; j < 2; ++j )
	{
		float rAx = L.an[j].x, rAy = L.an[j].y, rBx = L.an[j].z, rBy = L.an[j].w;
		float rsAx = A.dqc * rAx - A.dqs * rAy;
		float rsAy = A.dqs * rAx + A.dqc * rAy;
		float rsBx = B.dqc * rBx - B.dqs * rBy;
		float rsBy = B.dqs * rBx + B.dqc * rBy;
		float dsx = dpx + ( rsBx - rsAx );
		float dsy = dpy + ( rsBy - rsAy );
		float s = ( nm.x * dsx + nm.y * dsy ) + L.pt[j].x;
		bool mask = s > 0.0f;
		float specBias = s * inv_h;
		float softBias = lmax( biasRate * s, minBiasVel );
		float bias = mask ? specBias : softBias;
		float pointMassScale = mask ? 1.0f : massScale;
		float pointImpulseScale = mask ? 0.0f : impulseScale;
		float dvx = ( B.vx - B.w * rBy ) - ( A.vx - A.w * rAy );
		float dvy = ( B.vy + B.w * rBx ) - ( A.vy + A.w * rAx );
		float vn = dvx * nm.x + dvy * nm.y;
		float negImpulse = L.pt[j].y * ( pointMassScale * ( vn + bias ) ) + pointImpulseScale * nis[j];
		float newImpulse = lmax( nis[j] - negImpulse, 0.0f );
		float impulse = newImpulse - nis[j];
		nis[j] = newImpulse;
		tots[j] = tots[j] + newImpulse;
		totalNormalImpulse = totalNormalImpulse + newImpulse;
		float Px = impulse * nm.x;
		float Py = impulse * nm.y;
		A.vx = A.vx - ms.x * Px;
		A.vy = A.vy - ms.x * Py;
		A.w = A.w - ms.y * ( rAx * Py - rAy * Px );
		B.vx = B.vx + ms.z * Px;
		B.vy = B.vy + ms.z * Py;
		B.w = B.w + ms.w * ( rBx * Py - rBy * Px );
	}
	float tx = nm.y;
	float ty = 0.0f - nm.x;
	for ( int j = 0; j < 2; ++j )
	{
		float rAx = L.an[j].x, rAy = L.an[j].y, rBx = L.an[j].z, rBy = L.an[j].w;
		float dvx = ( B.vx - B.w * rBy ) - ( A.vx - A.w * rAy );
		float dvy = ( B.vy + B.w * rBx ) - ( A.vy + A.w * rAx );
		float vt = dvx * tx + dvy * ty;
		vt = vt - nm.w;
		float negImpulse = L.pt[j].z * vt;
		float maxFriction = nm.z * nis[j];
		float newImpulse = tis[j] - negImpulse;
		newImpulse = lmax( 0.0f - maxFriction, lmin( newImpulse, maxFriction ) );
		float impulse = newImpulse - tis[j];
		tis[j] = newImpulse;
		float Px = impulse * tx;
		float Py = impulse * ty;
		A.vx = A.vx - ms.x * Px;
		A.vy = A.vy - ms.x * Py;
		A.w = A.w - ms.y * ( rAx * Py - rAy * Px );
		B.vx = B.vx + ms.z * Px;
		B.vy = B.vy + ms.z * Py;
		B.w = B.w + ms.w * ( rBx * Py - rBy * Px );
	}
	{
		float deltaLambda = misc.z * ( A.w - B.w );
		float lambda = misc.w;
		float maxLambda = misc.y * totalNormalImpulse;
		float nb = -maxLambda;
		float r = lmax( nb, lmin( lambda + deltaLambda, maxLambda ) );
		misc.w = r;
		deltaLambda = r - lambda;
		A.w = A.w - ms.y * deltaLambda;
		B.w = B.w + ms.w * deltaLambda;
	}
	L.imp = make_float4( nis[0], nis[1], tis[0], tis[1] );
	L.tot = make_float4( tots[0], tots[1], 0.0f, 0.0f );
	L.misc = misc;
}

// contact_solver.c:1969-2076 (lanes with restitution 0 are unchanged)
__device__ __forceinline__ void lane_restitution( BState& A, BState& B, Lane& L, float threshold )
{
	float restitution = L.misc.x;
	if ( restitution == 0.0f )
		return;
	const float4 ms = L.ms, nm = L.nm;
	float nis[2] = { L.imp.x, L.imp.y };
	float tots[2] = { L.tot.x, L.tot.y };
	for ( int j = 0; j < 2; ++j )
	{
		bool mask1 = ( L.pt[j].w + threshold ) > 0.0f;
		bool mask2 = tots[j] == 0.0f;
		float mass = ( mask1 || mask2 ) ? 0.0f : L.pt[j].y;
		float rAx = L.an[j].x, rAy = L.an[j].y, rBx = L.an[j].z, rBy = L.an[j].w;
		float dvx = ( B.vx - B.w * rBy ) - ( A.vx - A.w * rAy );
		float dvy = ( B.vy + B.w * rBx ) - ( A.vy + A.w * rAx );
		float vn = dvx * nm.x + dvy * nm.y;
		float negImpulse = mass * ( vn + restitution * L.pt[j].w );
		float newImpulse = lmax( nis[j] - negImpulse, 0.0f );
		float impulse = newImpulse - nis[j];
		nis[j] = newImpulse;
		float Px = impulse * nm.x;
		float Py = impulse * nm.y;
		A.vx = A.vx - ms.x * Px;
		A.vy = A.vy - ms.x * Py;
		A.w = A.w - ms.y * ( rAx * Py - rAy * Px );
		B.vx = B.vx + ms.z * Px;
		B.vy = B.vy + ms.z * Py;
		B.w = B.w + ms.w * ( rBx * Py - rBy * Px );
	}
	L.imp.x = nis[0];
	L.imp.y = nis[1];
}

// contact_solver.c:160-225
__device__ __forceinline__ void warm_overflow( BState& A, BState& B, const Lane& L, int count )
{
	float4 ms = L.ms, nm = L.nm, imp = L.imp;
	fv2 normal = mk( nm.x, nm.y );
	fv2 tangent = vright( normal );
	fv2 vA = mk( A.vx, A.vy ), vB = mk( B.vx, B.vy );
	float wA = A.w, wB = B.w;
	float nis[2] = { imp.x, imp.y };
	float tis[2] = { imp.z, imp.w };
#pragma unroll
	for ( int j = 0; j < 2; ++j )
	{
		if ( j >= count )
			break;
		fv2 rA = mk( L.an[j].x, L.an[j].y ), rB = mk( L.an[j].z, L.an[j].w );
		fv2 P = vadd( vscale( nis[j], normal ), vscale( tis[j], tangent ) );
		wA -= ms.y * vcross( rA, P );
		vA = vmuladd( vA, -ms.x, P );
		wB += ms.w * vcross( rB, P );
		vB = vmuladd( vB, ms.z, P );
	}
	wA -= ms.y * L.misc.w;
	wB += ms.w * L.misc.w;
	A.vx = vA.x;
	A.vy = vA.y;
	A.w = wA;
	B.vx = vB.x;
	B.vy = vB.y;
	B.w = wB;
}

// contact_solver.c:227-380
__device__ __forceinline__ void solve_overflow( BState& A, BState& B, Lane& L, int count, Soft soft, float inv_h,
												float pushout, bool useBias )
{
	float4 ms = L.ms;
	float mA = ms.x, iA = ms.y, mB = ms.z, iB = ms.w;
	float4 nm = L.nm;
	float4 misc = L.misc;
	fv2 vA = mk( A.vx, A.vy ), vB = mk( B.vx, B.vy );
	float wA = A.w, wB = B.w;
	frot dqA, dqB;
	dqA.c = A.dqc;
	dqA.s = A.dqs;
	dqB.c = B.dqc;
	dqB.s = B.dqs;
	fv2 dp = vsub( mk( B.dpx, B.dpy ), mk( A.dpx, A.dpy ) );
	fv2 normal = mk( nm.x, nm.y );
	fv2 tangent = vright( normal );
	float friction = nm.z;
	float totalNormalImpulse = 0.0f;
	float nis[2] = { L.imp.x, L.imp.y };
	float tis[2] = { L.imp.z, L.imp.w };
	float tots[2] = { L.tot.x, L.tot.y };
#pragma unroll
	for ( int j = 0; j < 2; ++j )
	{
		if ( j >= count )
			break;
		fv2 rA = mk( L.an[j].x, L.an[j].y ), rB = mk( L.an[j].z, L.an[j].w );
		fv2 ds = vadd( dp, vsub( rrot( dqB, rB ), rrot( dqA, rA ) ) );
		float s = L.pt[j].x + vdot( ds, normal );
		float velocityBias = 0.0f;
		float massScale = 1.0f;
		float impulseScale = 0.0f;
		if ( s > 0.0f )
			velocityBias = s * inv_h;
		else if ( useBias )
		{
			velocityBias = fmax_s( soft.biasRate * s, -pushout );
			massScale = soft.massScale;
			impulseScale = soft.impulseScale;
		}
		fv2 vrA = vadd( vA, vcrossSV( wA, rA ) );
		fv2 vrB = vadd( vB, vcrossSV( wB, rB ) );
		float vn = vdot( vsub( vrB, vrA ), normal );
		float impulse = -L.pt[j].y * massScale * ( vn + velocityBias ) - impulseScale * nis[j];
		float newImpulse = fmax_s( nis[j] + impulse, 0.0f );
		impulse = newImpulse - nis[j];
		nis[j] = newImpulse;
		tots[j] += newImpulse;
		totalNormalImpulse += newImpulse;
		fv2 P = vscale( impulse, normal );
		vA = vmulsub( vA, mA, P );
		wA -= iA * vcross( rA, P );
		vB = vmuladd( vB, mB, P );
		wB += iB * vcross( rB, P );
	}
#pragma unroll
	for ( int j = 0; j < 2; ++j )
	{
		if ( j >= count )
			break;
		fv2 rA = mk( L.an[j].x, L.an[j].y ), rB = mk( L.an[j].z, L.an[j].w );
		fv2 vrB = vadd( vB, vcrossSV( wB, rB ) );
		fv2 vrA = vadd( vA, vcrossSV( wA, rA ) );
		float vt = vdot( vsub( vrB, vrA ), tangent ) - nm.w;
		float impulse = L.pt[j].z * ( -vt );
		float maxFriction = friction * nis[j];
		float newImpulse = fclamp_s( tis[j] + impulse, -maxFriction, maxFriction );
		impulse = newImpulse - tis[j];
		tis[j] = newImpulse;
		fv2 P = vscale( impulse, tangent );
		vA = vmulsub( vA, mA, P );
		wA -= iA * vcross( rA, P );
		vB = vmuladd( vB, mB, P );
		wB += iB * vcross( rB, P );
	}
	{
		float deltaLambda = -misc.z * ( wB - wA );
		float lambda = misc.w;
		float maxLambda = misc.y * totalNormalImpulse;
		misc.w = fclamp_s( lambda + deltaLambda, -maxLambda, maxLambda );
		deltaLambda = misc.w - lambda;
		wA -= iA * deltaLambda;
		wB += iB * deltaLambda;
	}
	L.imp = make_float4( nis[0], nis[1], tis[0], tis[1] );
	L.tot = make_float4( tots[0], tots[1], 0.0f, 0.0f );
	L.misc = misc;
	A.vx = vA.x;
	A.vy = vA.y;
	A.w = wA;
	B.vx = vB.x;
	B.vy = vB.y;
	B.w = wB;
}

// contact_solver.c:382-478
__device__ __forceinline__ void restitution_overflow( BState& A, BState& B, Lane& L, int count, float threshold )
{
	float restitution = L.misc.x;
	if ( restitution == 0.0f )
		return;
	float4 ms = L.ms;
	float mA = ms.x, iA = ms.y, mB = ms.z, iB = ms.w;
	fv2 vA = mk( A.vx, A.vy ), vB = mk( B.vx, B.vy );
	float wA = A.w, wB = B.w;
	fv2 normal = mk( L.nm.x, L.nm.y );
	float nis[2] = { L.imp.x, L.imp.y };
	float tots[2] = { L.tot.x, L.tot.y };
#pragma unroll
	for ( int j = 0; j < 2; ++j )
	{
		if ( j >= count )
			break;
		if ( L.pt[j].w > -threshold || tots[j] == 0.0f )
			continue;
		fv2 rA = mk( L.an[j].x, L.an[j].y ), rB = mk( L.an[j].z, L.an[j].w );
		fv2 vrB = vadd( vB, vcrossSV( wB, rB ) );
		fv2 vrA = vadd( vA, vcrossSV( wA, rA ) );
		float vn = vdot( vsub( vrB, vrA ), normal );
		float impulse = -L.pt[j].y * ( vn + restitution * L.pt[j].w );
		float newImpulse = fmax_s( nis[j] + impulse, 0.0f );
		impulse = newImpulse - nis[j];
		nis[j] = newImpulse;
		tots[j] += impulse;
		fv2 P = vscale( impulse, normal );
		vA = vmulsub( vA, mA, P );
		wA -= iA * vcross( rA, P );
		vB = vmuladd( vB, mB, P );
		wB += iB * vcross( rB, P );
	}
	L.imp.x = nis[0];
	L.imp.y = nis[1];
	L.tot.x = tots[0];
	L.tot.y = tots[1];
	A.vx = vA.x;
	A.vy = vA.y;
	A.w = wA;
	B.vx = vB.x;
	B.vy = vB.y;
	B.w = wB;
}
