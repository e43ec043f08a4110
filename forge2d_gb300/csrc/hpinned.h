// Page-locked arrays of the host's trees.
#pragma once

#include <cuda_runtime.h>

#include <cstdlib>
#include <new>
#include <vector>

// Page-locked arrays from PINNED_BYTES up (a tree of 4096 nodes): a tree is
// edited on the host between two steps, so its arrays go both ways every time.
// From pageable memory the 3.4 MB of a 20k-body world's tree took some 450 us
// each way. Below, and without a device, plain memory.
#define PINNED_BYTES 65536
// A long array's block starts with how it was allocated: cudaFreeHost also
// fails on page-locked blocks, after a device error or as the process ends,
// and such a block is none of the heap's.
#define PINNED_HEAD 64
template <typename T> struct PinnedAlloc
{
	typedef T value_type;
	PinnedAlloc() = default;
	template <typename U> PinnedAlloc( const PinnedAlloc<U>& ) {}
	T* allocate( size_t n )
	{
		const bool head = n * sizeof( T ) >= PINNED_BYTES;
		void* p = nullptr;
		const size_t bytes = n * sizeof( T ) + ( head ? PINNED_HEAD : 0 );
		bool locked = false;
		if ( head )
		{
			locked = cudaMallocHost( &p, bytes ) == cudaSuccess;
			if ( !locked )
				cudaGetLastError();
		}
		if ( !locked )
			p = malloc( bytes );
		if ( p == nullptr )
			throw std::bad_alloc();
		if ( !head )
			return (T*)p;
		*(bool*)p = locked;
		return (T*)( (char*)p + PINNED_HEAD );
	}
	void deallocate( T* p, size_t n )
	{
		if ( n * sizeof( T ) < PINNED_BYTES )
		{
			free( p );
			return;
		}
		void* block = (char*)p - PINNED_HEAD;
		if ( !*(bool*)block )
			free( block );
		else if ( cudaFreeHost( block ) != cudaSuccess )
			cudaGetLastError(); // left to the process's end
	}
	template <typename U> bool operator==( const PinnedAlloc<U>& ) const { return true; }
	template <typename U> bool operator!=( const PinnedAlloc<U>& ) const { return false; }
};
template <typename T> using PinnedVector = std::vector<T, PinnedAlloc<T>>;
