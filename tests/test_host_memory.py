"""Host memory of the library against a fake of the CUDA allocation calls that
fails where it is told to: no GPU, no driver."""
from __future__ import annotations

import os
import re
import shutil
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "forge2d_gb300", "csrc")

FAKE = r"""
#include <cuda_runtime.h>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <set>

// every call counts; call number `failAt` fails (1: the first)
static int calls = 0, failAt = 0, sets = 0, bad = 0;
static std::set<void*> live;
static void* fixedBlock = nullptr; // given instead of heap memory, and not taken back
static bool fails() { calls += 1; return calls == failAt; }
static cudaError_t give( void** p, size_t n )
{
	if ( fails() )
		return cudaErrorMemoryAllocation; // *p stays as it was
	if ( fixedBlock )
	{
		*p = fixedBlock;
		return cudaSuccess;
	}
	*p = malloc( n );
	live.insert( *p );
	return cudaSuccess;
}
static cudaError_t take( void* p )
{
	if ( live.erase( p ) == 0 )
	{
		bad += 1;
		return cudaErrorInvalidValue;
	}
	free( p );
	return cudaSuccess;
}
extern "C" cudaError_t cudaMalloc( void** p, size_t n ) { return give( p, n ); }
extern "C" cudaError_t cudaMallocHost( void** p, size_t n ) { return give( p, n ); }
extern "C" cudaError_t cudaFree( void* p ) { return take( p ); }
extern "C" cudaError_t cudaFreeHost( void* p ) { return take( p ); }
extern "C" cudaError_t cudaMemsetAsync( void* p, int v, size_t n, cudaStream_t ) { sets += 1; memset( p, v, n ); return cudaSuccess; }
#define CHECK( x ) do { if ( !( x ) ) { printf( "line %d: %s\n", __LINE__, #x ); return 1; } } while ( 0 )
"""

QUERY = FAKE + r"""
#include "hscratch.h"
int main()
{
	// the allocation that fails: best, count, ray, found, ids; 6: none
	for ( int k = 1; k <= 6; ++k )
	{
		calls = 0;
		failAt = k;
		sets = 0;
		QueryScratch q;
		CHECK( q.ready( 10, nullptr ) == ( k == 6 ) );
		failAt = 0;
		CHECK( q.ready( 10, nullptr ) );
		CHECK( q.best && q.count && q.ray && q.found && q.ids && q.idCap >= 10 );
		CHECK( *q.best == ~0ull && q.count[0] == 0 && q.count[1] == 0 && sets == 2 );
		CHECK( live.size() == 5 );
		// a list that cannot grow is asked for again
		failAt = calls + 1;
		CHECK( !q.ready( 5000, nullptr ) );
		failAt = 0;
		CHECK( q.ready( 5000, nullptr ) && q.ids && q.idCap >= 5000 );
		q.release();
		CHECK( live.empty() && bad == 0 );
	}
	return 0;
}
"""

PINNED = FAKE.replace("static cudaError_t give", r"""
static int errors = 0; // reads of the last error
extern "C" cudaError_t cudaGetLastError() { errors += 1; return cudaSuccess; }
static cudaError_t give""") + r"""
#include "hpinned.h"
struct F4 { float x, y, z, w; };
template <typename T> static int arrays()
{
	const size_t sizes[] = { 1, 64, PINNED_BYTES / sizeof( T ) - 1, PINNED_BYTES / sizeof( T ), 100000 };
	for ( size_t n : sizes )
		for ( int refused = 0; refused < 2; ++refused )
		{
			calls = 0;
			failAt = refused;
			{
				PinnedVector<T> v( n );
				CHECK( ( (size_t)v.data() & 15 ) == 0 );
				CHECK( live.size() == ( n * sizeof( T ) >= PINNED_BYTES && !refused ? 1u : 0u ) );
				memset( (void*)v.data(), 0x5a, n * sizeof( T ) );
				PinnedVector<T> u = v;
				u.resize( 2 * n );
				CHECK( memcmp( u.data(), v.data(), n * sizeof( T ) ) == 0 );
				v = std::move( u );
			}
			CHECK( live.empty() && bad == 0 );
		}
	return 0;
}
int main()
{
	CHECK( arrays<int>() == 0 && arrays<F4>() == 0 && arrays<unsigned long long>() == 0 );
	// a page-locked block that cannot be given back: not the heap's
	static char locked[PINNED_BYTES + 4096];
	char* at = locked + 64 - ( (size_t)locked & 63 );
	fixedBlock = at;
	{
		PinnedVector<int> v( PINNED_BYTES / sizeof( int ) );
		CHECK( (char*)v.data() >= at && (char*)( v.data() + v.size() ) <= at + PINNED_BYTES + 1024 );
	}
	CHECK( bad == 1 );
	return 0;
}
"""

LAST_ERROR = PINNED[:PINNED.index("int main()")] + r"""
int main()
{
	{
		PinnedVector<int> small( 100 ), large( PINNED_BYTES );
	}
	CHECK( errors == 0 ); // an error of another call waits for who asks for it
	calls = 0;
	failAt = 1;
	PinnedVector<int> refused( PINNED_BYTES );
	CHECK( errors == 1 );
	return 0;
}
"""


def _run(tmp_path, name, source):
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"))), "include")
    path = tmp_path / (name + ".cpp")
    path.write_text(source)
    exe = str(tmp_path / name)
    r = subprocess.run(["g++", "-std=c++17", "-O1", "-I" + CSRC, "-I" + cuda, str(path), "-o", exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, (r.returncode, r.stdout + r.stderr)


def test_query_workspace_survives_failing_allocations(tmp_path):
    _run(tmp_path, "query", QUERY)


def test_page_locked_blocks_are_not_the_heaps(tmp_path):
    _run(tmp_path, "pinned", PINNED)


def test_other_calls_errors_are_kept(tmp_path):
    _run(tmp_path, "last_error", LAST_ERROR)


def test_world_memory_is_written_in_stream_order():
    """A world's streams do not wait for the default stream: clears of and
    copies to its device memory go through its own, or a step may run ahead
    of them (synchronous copies to the host follow a wait)."""
    source = open(os.path.join(CSRC, "world.cu")).read()
    assert re.findall(r"\bcudaMemset\(", source) == []
    copies = re.findall(r"\bcudaMemcpy\((?:[^;]*?)\);", source, re.S)
    assert copies and [c for c in copies if "cudaMemcpyDeviceToHost" not in c] == []


def test_model_edits_end_with_a_wait():
    """A world may read a model on its own stream right after its edit."""
    source = open(os.path.join(CSRC, "mlp.cu")).read()
    for name in ("f2d_mlp_create", "f2d_mlp_set_params", "f2d_mlp_set_normalization"):
        body = source[source.index(" " + name + "("):]
        assert "cudaDeviceSynchronize()" in body[:body.index("\n}\n")], name
