// Single rows from the host by value.
//
// A body has fourteen device arrays and a shape twelve; a copy each is some
// 4 us of host time, so a body created or edited between two steps cost about
// 110 us in copies alone. Up to ROW_BATCH rows travel in the arguments of one
// launch instead (no staging memory to keep or to wait for). Ranges of more
// than ROWS_BY_VALUE rows, a level's load, stay one copy per array: there a
// copy moves thousands of rows at the link's rate.
#include "dworld.cuh"
#include "kernels.cuh"

__global__ void k_body_rows( DWorld w, BodyRows rows )
{
	if ( (int)threadIdx.x >= rows.n )
		return;
	const BodyRow& r = rows.row[threadIdx.x];
	const int b = r.id;
	w.xf[b] = r.xf;
	w.vel[b] = r.vel;
	w.delta[b] = r.delta;
	w.center[b] = r.center;
	w.sweep0[b] = r.sweep0;
	w.localCenter[b] = r.localCenter;
	w.massv[b] = r.massv;
	w.damp[b] = r.damp;
	w.bodyGravity[b] = r.gravity;
	w.force[b] = r.force;
	w.bflags[b] = r.flags;
	w.headShape[b] = r.headShape;
	w.headJoint[b] = r.headJoint;
	w.jointCountB[b] = r.jointCount;
}

__global__ void k_shape_rows( DWorld w, ShapeRows rows )
{
	if ( (int)threadIdx.x >= rows.n )
		return;
	const ShapeRow& r = rows.row[threadIdx.x];
	const int s = r.id;
	for ( int k = 0; k < GEOM_F4; ++k )
		w.geom[(size_t)s * GEOM_F4 + k] = r.geom[k];
	w.aabb[s] = r.aabb;
	w.fat[s] = r.fat;
	w.mat[s] = r.mat;
	w.cat[s] = r.cat;
	w.mask[s] = r.mask;
	w.group[s] = r.group;
	w.shapeBody[s] = r.body;
	w.shapeSub[s] = r.sub;
	w.sflags[s] = r.flags;
	w.proxyKey[s] = r.proxyKey;
	w.nextShape[s] = r.next;
}

// Few buffered proxies join the move array, in their order (what the step's
// host-move chain does for any number of them).
__global__ void k_few_moves( DWorld w, FewMoves m )
{
	const int lane = threadIdx.x;
	const int s = lane < m.n ? m.shape[lane] : 0;
	const int f = lane < m.n ? w.sflags[s] : 0;
	const bool joins = ( f & ( SF_USED | SF_PROXY | SF_MOVED ) ) == ( SF_USED | SF_PROXY );
	const unsigned mask = __ballot_sync( 0xffffffffu, joins );
	const int base = w.sc->moveArrayCount;
	__syncwarp();
	if ( joins )
	{
		const int slot = base + __popc( mask & ( ( 1u << lane ) - 1u ) );
		w.moveShape[slot] = s;
		w.shapeMove[s] = slot;
		w.sflags[s] = f | SF_MOVED;
	}
	if ( lane == 0 )
		w.sc->moveArrayCount = base + __popc( mask );
}

void launch_body_rows( DWorld& w, const BodyRows& rows, cudaStream_t st )
{
	k_body_rows<<<1, 32, 0, st>>>( w, rows );
}

void launch_shape_rows( DWorld& w, const ShapeRows& rows, cudaStream_t st )
{
	k_shape_rows<<<1, 32, 0, st>>>( w, rows );
}

void launch_few_moves( DWorld& w, const FewMoves& moves, cudaStream_t st )
{
	k_few_moves<<<1, 32, 0, st>>>( w, moves );
}
