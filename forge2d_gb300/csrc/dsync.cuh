// Device-wide synchronisation primitives shared by the persistent kernels.
//
// grid_barrier: for cooperative launches only (co-residency of every block
// is guaranteed by cudaLaunchCooperativeKernel). One monotonically
// increasing arrival counter, zeroed on the stream before the launch:
// barrier number e is passed when the counter reaches e x gridDim.x. Thread 0
// of each block publishes the block's writes with a release add and waits
// with acquire loads; __syncthreads orders the rest of the block on either
// side. Shared data written before a barrier is read after it with L2 (.cg)
// or acquire loads, so no stale L1 line survives. Every wait is bounded: a
// block that gives up sets the timeout bit in *err and every other block
// leaves at its next poll of that word.
#pragma once

#include <cuda_runtime.h>

#define F2D_SPIN_LIMIT ( 1ll << 24 )
#define F2D_ERR_BARRIER_TIMEOUT 0x4

__device__ __forceinline__ void red_release_add( unsigned* p, unsigned v )
{
	asm volatile( "red.release.gpu.global.add.u32 [%0], %1;" ::"l"( p ), "r"( v ) : "memory" );
}

__device__ __forceinline__ unsigned ld_acquire_u32( const unsigned* p )
{
	unsigned v;
	asm volatile( "ld.acquire.gpu.global.u32 %0, [%1];" : "=r"( v ) : "l"( p ) : "memory" );
	return v;
}

__device__ __forceinline__ unsigned long long ld_acquire_u64( const unsigned long long* p )
{
	unsigned long long v;
	asm volatile( "ld.acquire.gpu.global.u64 %0, [%1];" : "=l"( v ) : "l"( p ) : "memory" );
	return v;
}

__device__ __forceinline__ void st_release_u64( unsigned long long* p, unsigned long long v )
{
	asm volatile( "st.release.gpu.global.u64 [%0], %1;" ::"l"( p ), "l"( v ) : "memory" );
}

__device__ __forceinline__ int ld_relaxed_s32( const int* p )
{
	int v;
	asm volatile( "ld.relaxed.gpu.global.s32 %0, [%1];" : "=r"( v ) : "l"( p ) : "memory" );
	return v;
}

// counter: zeroed before the launch; epoch: barriers this block has passed
// in this launch (identical on every block). Returns false on timeout.
__device__ __forceinline__ bool grid_barrier( unsigned* counter, int* err, unsigned& epoch )
{
	__shared__ int s_timedOut;
	__syncthreads();
	epoch += 1;
	if ( threadIdx.x == 0 )
	{
		unsigned target = epoch * gridDim.x;
		red_release_add( counter, 1u );
		long long spins = 0;
		int timedOut = 0;
		while ( (int)( ld_acquire_u32( counter ) - target ) < 0 )
		{
			++spins;
			if ( spins > F2D_SPIN_LIMIT ||
				 ( ( spins & 1023 ) == 0 && ( ld_relaxed_s32( err ) & F2D_ERR_BARRIER_TIMEOUT ) ) )
			{
				atomicOr( err, F2D_ERR_BARRIER_TIMEOUT );
				timedOut = 1;
				break;
			}
		}
		s_timedOut = timedOut;
	}
	__syncthreads();
	return s_timedOut == 0;
}

// Decoupled look-back over tiles claimed in launch order, one word per tile
// (zeroed before the launch): flag << 32 | value, 1 aggregate, 2 inclusive
// prefix. A tile publishes its aggregate, then one whole warp asks for its
// exclusive prefix, 32 preceding tiles at a time (a lane per word alone would
// pay an L2 round trip per tile).
__device__ __forceinline__ void lookback_publish( unsigned long long* state, int tile, int aggregate )
{
	st_release_u64( state + tile, ( tile == 0 ? 2ull << 32 : 1ull << 32 ) | (unsigned)aggregate );
}

__device__ __forceinline__ int lookback_prefix( unsigned long long* state, int tile, int aggregate, int* err )
{
	const int lane = threadIdx.x & 31;
	int prefix = 0;
	for ( int end = tile; end > 0; end -= 32 )
	{
		const int j = end - 1 - lane;
		unsigned long long v = 2ull << 32;
		for ( long long spins = 0; j >= 0; )
		{
			v = ld_acquire_u64( state + j );
			if ( ( v >> 32 ) != 0ull )
				break;
			if ( ++spins > F2D_SPIN_LIMIT )
			{
				atomicOr( err, F2D_ERR_BARRIER_TIMEOUT );
				v = 2ull << 32;
				break;
			}
		}
		__syncwarp();
		const unsigned done = __ballot_sync( 0xffffffffu, ( v >> 32 ) == 2ull );
		const int last = done ? __ffs( done ) - 1 : 31;
		prefix += __reduce_add_sync( 0xffffffffu, lane <= last ? (int)(unsigned)( v & 0xffffffffull ) : 0 );
		if ( done )
			break;
	}
	if ( lane == 0 && tile > 0 )
		st_release_u64( state + tile, ( 2ull << 32 ) | (unsigned)( prefix + aggregate ) );
	return prefix;
}
