// A world's workspace for ray and box queries: allocated once, guarded for
// calls from several threads, freed with the world.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <mutex>

#define QUERY_HOST_IDS 2048 // ids that reach the host without a copy of their own
struct QueryScratch
{
	std::mutex lock;
	unsigned long long* best = nullptr; // closest ray: fraction bits << 32 | shape; ~0 between calls
	int* count = nullptr;				// blocks done, hits; 0 between calls
	int* ids = nullptr;					// device: every hit of a box query
	int idCap = 0;
	float* ray = nullptr;	 // pinned, written by the kernel
	int* found = nullptr;	 // pinned: hits, then up to QUERY_HOST_IDS ids
	bool whole = false;		 // all but the id list is there and set up

	// The workspace with an id list for `shapes` (the caller holds the lock).
	// False when an allocation fails: what it needs is then tried again by the
	// next call.
	bool ready( int shapes, cudaStream_t st )
	{
		if ( !whole )
		{
			if ( cudaMalloc( (void**)&best, sizeof( unsigned long long ) ) != cudaSuccess ||
				 cudaMalloc( (void**)&count, 2 * sizeof( int ) ) != cudaSuccess ||
				 cudaMallocHost( (void**)&ray, 8 * sizeof( float ) ) != cudaSuccess ||
				 cudaMallocHost( (void**)&found, ( 1 + QUERY_HOST_IDS ) * sizeof( int ) ) != cudaSuccess )
			{
				release();
				return false;
			}
			cudaMemsetAsync( best, 0xff, sizeof( unsigned long long ), st );
			cudaMemsetAsync( count, 0, 2 * sizeof( int ), st );
			whole = true;
		}
		if ( shapes > idCap )
		{
			drop( ids );
			idCap = 0;
			int cap = std::max( 1024, 2 * shapes );
			if ( cudaMalloc( (void**)&ids, sizeof( int ) * (size_t)cap ) != cudaSuccess )
			{
				ids = nullptr;
				return false;
			}
			idCap = cap;
		}
		return true;
	}

	void release()
	{
		drop( best );
		drop( count );
		drop( ids );
		idCap = 0;
		if ( ray )
			cudaFreeHost( ray );
		if ( found )
			cudaFreeHost( found );
		ray = nullptr;
		found = nullptr;
		whole = false;
	}

  private:
	template <typename T> static void drop( T*& p )
	{
		if ( p )
			cudaFree( p );
		p = nullptr;
	}
};
