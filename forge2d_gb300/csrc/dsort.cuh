// One-launch device sort and scan for the world step.
//
// Element counts live in device memory (the step is enqueued without host
// round trips), so the launch shapes are fixed and each kernel reads n
// itself.
//
// * sort_coop: stable LSD radix sort of (key, value) rows by the low `bits`
//   bits of the key. Up to CSORT_SMALL rows block 0 sorts alone in shared
//   memory (bitonic on (key, value), which is the same order the stable sort
//   gives when the input values ascend); up to BSORT_MAX rows, one block with
//   the rows in registers (k_sort_block); above that, ONE cooperative launch (k_sort_coop):
//   per 8-bit digit, a block histogram, a grid barrier, per-block digit
//   offsets, a stable scatter (warp match_any ranks) and another grid barrier.
// * scan_lookback: exclusive scan of n ints in one launch (decoupled
//   look-back across tiles claimed in launch order).
#pragma once

#include "dscan.cuh"
#include "dsync.cuh"
#include "dworld.cuh"

#include <climits>

#define CSORT_THREADS 1024
#define CSORT_SMALL 2048
#define CSORT_MAX_BLOCKS 256
#define SORT_LARGE_WORLD 4096 // shapes
#define CSORT_WARPS ( CSORT_THREADS / 32 )

#define LB_THREADS 1024
#define LB_ITEMS 8
#define LB_TILE ( LB_THREADS * LB_ITEMS )
#define LB_FLAG_AGG 1ull
#define LB_FLAG_PREFIX 2ull

template <typename K> __device__ __forceinline__ bool kv_less( K ka, int va, K kb, int vb )
{
	return ka < kb || ( ka == kb && va < vb );
}

// Optional last step of a sort: made[r] = lookup[key of row r >> shift].
struct SortDecode
{
	int* made;
	const int* lookup;
	int shift;
};

// One block's sort of up to BSORT_MAX rows. Bound by its chain of passes, not
// by memory (98 KB of keys at most): LSD radix, the rows in registers,
// BSORT_ITEMS a thread, exchanged through shared memory. The cooperative
// sort's passes pay two grid barriers and several L2 round trips each (100k
// pile's pair sort at its dense frames, caches cold: 48 -> 38 us). The limit is what shared memory holds of 64-bit keys.
#define BSORT_ITEMS 12
#define BSORT_MAX ( BSORT_ITEMS * CSORT_THREADS )

struct BSortSmem
{
	struct
	{
		unsigned long long key[BSORT_MAX];
		unsigned short row[BSORT_MAX];
		unsigned hist[CSORT_WARPS][256]; // per-warp digit counts, then first positions
		unsigned part[4][256];
		unsigned start[256];
		int scan[32];
		unsigned long long any, all;
	} radix;
};

template <typename K>
__global__ void __launch_bounds__( CSORT_THREADS, 1 )
	k_sort_block( K* keys, int* vals, const int* nPtr, int cap, int bits, const int* enable, SortDecode dec )
{
	extern __shared__ __align__( 16 ) unsigned char bsortRaw[];
	BSortSmem& sm = *reinterpret_cast<BSortSmem*>( bsortRaw );
	const int tid = threadIdx.x;
	if ( enable && *enable == 0 )
		return;
	const int n = min( *nPtr, cap );
	if ( n <= CSORT_SMALL || n > BSORT_MAX )
		return;
	const int lane = tid & 31, warp = tid >> 5;
	const int items = ( n + CSORT_THREADS - 1 ) / CSORT_THREADS;
	const int first = warp * items * 32 + lane; // the thread's rows: first + 32 * item
	K key[BSORT_ITEMS];
	unsigned tag[BSORT_ITEMS]; // original row | rank << 16
	unsigned long long any = 0ull, all = ~0ull;
#pragma unroll
	for ( int it = 0; it < BSORT_ITEMS; ++it )
	{
		const int r = first + 32 * it;
		const bool valid = it < items && r < n;
		key[it] = valid ? keys[r] : (K)0;
		tag[it] = (unsigned)r;
		if ( valid )
		{
			any |= (unsigned long long)key[it];
			all &= (unsigned long long)key[it];
		}
	}
	// a digit that every row shares needs no pass
	if ( tid == 0 )
	{
		sm.radix.any = 0ull;
		sm.radix.all = ~0ull;
	}
#pragma unroll
	for ( int off = 16; off > 0; off >>= 1 )
	{
		any |= __shfl_xor_sync( 0xffffffffu, any, off );
		all &= __shfl_xor_sync( 0xffffffffu, all, off );
	}
	__syncthreads();
	if ( lane == 0 )
	{
		atomicOr( &sm.radix.any, any );
		atomicAnd( &sm.radix.all, all );
	}
	__syncthreads();
	const unsigned long long diff = sm.radix.any ^ sm.radix.all;
	for ( int shift = 0; shift < bits; shift += 8 )
	{
		if ( ( ( diff >> shift ) & 0xffull ) == 0ull )
			continue;
		for ( int d = lane; d < 256; d += 32 )
			sm.radix.hist[warp][d] = 0u;
		__syncwarp();
		// ranks within the warp's rows, in row order
#pragma unroll
		for ( int it = 0; it < BSORT_ITEMS; ++it )
		{
			if ( it >= items )
				break;
			const bool valid = first + 32 * it < n;
			const unsigned d = valid ? (unsigned)( ( key[it] >> shift ) & 0xff ) : 256u;
			const unsigned peers = __match_any_sync( 0xffffffffu, d );
			const int leader = __ffs( peers ) - 1;
			unsigned base = 0u;
			if ( valid && lane == leader )
			{
				base = sm.radix.hist[warp][d];
				sm.radix.hist[warp][d] = base + __popc( peers );
			}
			base = __shfl_sync( 0xffffffffu, base, leader );
			tag[it] = ( tag[it] & 0xffffu ) | ( ( base + __popc( peers & ( ( 1u << lane ) - 1u ) ) ) << 16 );
			__syncwarp();
		}
		__syncthreads();
		// first position of every (digit, warp)
		{
			const int d = tid & 255, q = tid >> 8;
			unsigned sum = 0u;
#pragma unroll
			for ( int k = 0; k < CSORT_WARPS / 4; ++k )
				sum += sm.radix.hist[q * ( CSORT_WARPS / 4 ) + k][d];
			sm.radix.part[q][d] = sum;
			__syncthreads();
			unsigned total = 0u;
			if ( tid < 256 )
				total = sm.radix.part[0][tid] + sm.radix.part[1][tid] + sm.radix.part[2][tid] + sm.radix.part[3][tid];
			int dummy;
			const int begin = block_exclusive_scan_1024( (int)total, sm.radix.scan, &dummy );
			if ( tid < 256 )
				sm.radix.start[tid] = (unsigned)begin;
			__syncthreads();
			unsigned run = sm.radix.start[d];
			for ( int k = 0; k < q; ++k )
				run += sm.radix.part[k][d];
#pragma unroll
			for ( int k = 0; k < CSORT_WARPS / 4; ++k )
			{
				unsigned* h = &sm.radix.hist[q * ( CSORT_WARPS / 4 ) + k][d];
				const unsigned v = *h;
				*h = run;
				run += v;
			}
		}
		__syncthreads();
#pragma unroll
		for ( int it = 0; it < BSORT_ITEMS; ++it )
			if ( it < items && first + 32 * it < n )
			{
				const unsigned dst = sm.radix.hist[warp][(unsigned)( ( key[it] >> shift ) & 0xff )] + ( tag[it] >> 16 );
				sm.radix.key[dst] = (unsigned long long)key[it];
				sm.radix.row[dst] = (unsigned short)tag[it];
			}
		__syncthreads();
#pragma unroll
		for ( int it = 0; it < BSORT_ITEMS; ++it )
		{
			const int r = first + 32 * it;
			if ( it < items && r < n )
			{
				key[it] = (K)sm.radix.key[r];
				tag[it] = sm.radix.row[r];
			}
		}
	}
	if ( vals )
	{
		// the values follow their rows: all read before any is written
#pragma unroll
		for ( int it = 0; it < BSORT_ITEMS; ++it )
			if ( it < items && first + 32 * it < n )
				tag[it] = (unsigned)__ldcg( vals + ( tag[it] & 0xffffu ) );
		__syncthreads();
	}
#pragma unroll
	for ( int it = 0; it < BSORT_ITEMS; ++it )
	{
		const int r = first + 32 * it;
		if ( it < items && r < n )
		{
			keys[r] = key[it];
			if ( vals )
				vals[r] = (int)tag[it];
			if ( dec.made )
				dec.made[r] = dec.lookup[key[it] >> dec.shift];
		}
	}
}

// shared memory of k_sort_coop: the bitonic buffers or the radix tables
union CSortSmem
{
	struct
	{
		unsigned long long key[CSORT_SMALL];
		int val[CSORT_SMALL];
	} small;
	struct
	{
		unsigned base[256];				   // running scatter base per digit
		unsigned warpHist[CSORT_WARPS][256]; // per-warp digit counts, then prefixes
		unsigned partTotal[4][256];		   // digit totals per quarter of the blocks
		unsigned partBefore[4][256];	   // same, only blocks before this one
		int scan[32];
	} radix;
};

template <typename K>
__global__ void __launch_bounds__( CSORT_THREADS )
	k_sort_coop( K* keys, int* vals, K* keysAlt, int* valsAlt, int* nPtr, int cap, int bits, unsigned* hist,
				 unsigned* counter, int* err, const int* enable, int skipUpTo, SortDecode dec )
{
	__shared__ CSortSmem sm;
	const int tid = threadIdx.x;
	if ( enable && *enable == 0 )
		return;
	const int n = min( *nPtr, cap );
	if ( n < 1 )
		return;
	// the count as it is kept
	if ( blockIdx.x == 0 && tid == 0 && *nPtr > n )
		*nPtr = n;
	if ( n <= CSORT_SMALL )
	{
		if ( blockIdx.x != 0 )
			return;
		int P = 2;
		while ( P < n )
			P <<= 1;
		for ( int i = tid; i < P; i += CSORT_THREADS )
		{
			sm.small.key[i] = i < n ? (unsigned long long)keys[i] : ~0ull;
			sm.small.val[i] = i < n ? ( vals ? vals[i] : i ) : INT_MAX;
		}
		__syncthreads();
		for ( int k = 2; k <= P; k <<= 1 )
		{
			for ( int j = k >> 1; j > 0; j >>= 1 )
			{
				for ( int t = tid; t < ( P >> 1 ); t += CSORT_THREADS )
				{
					int i = ( ( t & ~( j - 1 ) ) << 1 ) | ( t & ( j - 1 ) );
					int l = i + j;
					unsigned long long ki = sm.small.key[i], kl = sm.small.key[l];
					int vi = sm.small.val[i], vl = sm.small.val[l];
					bool up = ( i & k ) == 0;
					bool swap = up ? kv_less( kl, vl, ki, vi ) : kv_less( ki, vi, kl, vl );
					if ( swap )
					{
						sm.small.key[i] = kl;
						sm.small.key[l] = ki;
						sm.small.val[i] = vl;
						sm.small.val[l] = vi;
					}
				}
				__syncthreads();
			}
		}
		for ( int i = tid; i < n; i += CSORT_THREADS )
		{
			keys[i] = (K)sm.small.key[i];
			if ( vals )
				vals[i] = sm.small.val[i];
			if ( dec.made )
				dec.made[i] = dec.lookup[keys[i] >> dec.shift];
		}
		return;
	}
	if ( n <= skipUpTo )
		return;

	unsigned epoch = 0;
	const int G = gridDim.x;
	const int per = ( n + G - 1 ) / G;
	const int lo = min( n, blockIdx.x * per ), hi = min( n, lo + per );
	const int lane = tid & 31, warp = tid >> 5;
	const int passes = ( bits + 7 ) / 8;
	// A digit every row shares needs no pass (a stable pass over it keeps
	// the order): the OR and the AND of all keys, one word pair per block in
	// the histogram buffer's last rows, which the histograms of at most
	// CSORT_MAX_BLOCKS - 4 blocks never reach.
	unsigned long long diff = ~0ull;
	if ( G <= CSORT_MAX_BLOCKS - 4 )
	{
		__shared__ unsigned long long sOr, sAnd;
		unsigned long long o = 0ull, a = ~0ull;
		for ( int i = lo + tid; i < hi; i += CSORT_THREADS )
		{
			unsigned long long k = (unsigned long long)__ldcg( keys + i );
			o |= k;
			a &= k;
		}
#pragma unroll
		for ( int off = 16; off > 0; off >>= 1 )
		{
			o |= __shfl_xor_sync( 0xffffffffu, o, off );
			a &= __shfl_xor_sync( 0xffffffffu, a, off );
		}
		if ( tid == 0 )
		{
			sOr = 0ull;
			sAnd = ~0ull;
		}
		__syncthreads();
		if ( lane == 0 )
		{
			atomicOr( &sOr, o );
			atomicAnd( &sAnd, a );
		}
		__syncthreads();
		unsigned long long* part = (unsigned long long*)( hist + 256 * ( CSORT_MAX_BLOCKS - 4 ) );
		if ( tid == 0 )
		{
			__stcg( part + 2 * blockIdx.x, sOr );
			__stcg( part + 2 * blockIdx.x + 1, sAnd );
		}
		if ( !grid_barrier( counter, err, epoch ) )
			return;
		if ( tid == 0 )
		{
			sOr = 0ull;
			sAnd = ~0ull;
		}
		__syncthreads();
		o = 0ull;
		a = ~0ull;
		for ( int b = tid; b < G; b += CSORT_THREADS )
		{
			o |= __ldcg( part + 2 * b );
			a &= __ldcg( part + 2 * b + 1 );
		}
#pragma unroll
		for ( int off = 16; off > 0; off >>= 1 )
		{
			o |= __shfl_xor_sync( 0xffffffffu, o, off );
			a &= __shfl_xor_sync( 0xffffffffu, a, off );
		}
		if ( lane == 0 )
		{
			atomicOr( &sOr, o );
			atomicAnd( &sAnd, a );
		}
		__syncthreads();
		diff = sOr ^ sAnd;
	}
	K* kin = keys;
	int* vin = vals;
	K* kout = keysAlt;
	int* vout = valsAlt;
	int done = 0;
	for ( int p = 0; p < passes; ++p )
	{
		const int shift = 8 * p;
		if ( ( ( diff >> shift ) & 0xffull ) == 0ull )
			continue;
		done += 1;
		// 1. digit histogram of this block's rows
		if ( tid < 256 )
			sm.radix.base[tid] = 0;
		__syncthreads();
		for ( int i = lo + tid; i < hi; i += CSORT_THREADS )
			atomicAdd( sm.radix.base + (unsigned)( ( __ldcg( kin + i ) >> shift ) & 0xff ), 1u );
		__syncthreads();
		if ( tid < 256 )
			hist[blockIdx.x * 256 + tid] = sm.radix.base[tid];
		if ( !grid_barrier( counter, err, epoch ) )
			return;
		// 2. this block's first output position per digit: rows of smaller
		// digits anywhere plus rows of this digit in earlier blocks
		{
			int d = tid & 255, q = tid >> 8;
			unsigned total = 0, before = 0;
			for ( int b = q; b < G; b += 4 )
			{
				unsigned v = __ldcg( hist + b * 256 + d );
				total += v;
				before += b < (int)blockIdx.x ? v : 0u;
			}
			sm.radix.partTotal[q][d] = total;
			sm.radix.partBefore[q][d] = before;
		}
		__syncthreads();
		unsigned digitTotal = 0, digitBefore = 0;
		if ( tid < 256 )
		{
			for ( int q = 0; q < 4; ++q )
			{
				digitTotal += sm.radix.partTotal[q][tid];
				digitBefore += sm.radix.partBefore[q][tid];
			}
		}
		int dummy;
		int digitStart = block_exclusive_scan_1024( (int)digitTotal, sm.radix.scan, &dummy );
		if ( tid < 256 )
			sm.radix.base[tid] = (unsigned)digitStart + digitBefore;
		__syncthreads();
		// 3. stable scatter, chunk by chunk in row order
		for ( int c0 = lo; c0 < hi; c0 += CSORT_THREADS )
		{
			int i = c0 + tid;
			bool valid = i < hi;
			K key = valid ? __ldcg( kin + i ) : (K)0;
			int val = ( valid && vin ) ? __ldcg( vin + i ) : 0;
			unsigned d = valid ? (unsigned)( ( key >> shift ) & 0xff ) : ( 256u + (unsigned)lane );
			for ( int k = tid; k < CSORT_WARPS * 256; k += CSORT_THREADS )
				( &sm.radix.warpHist[0][0] )[k] = 0;
			__syncthreads();
			unsigned peers = __match_any_sync( 0xffffffffu, d );
			unsigned rank = __popc( peers & ( ( 1u << lane ) - 1u ) );
			if ( valid && rank == 0 )
				sm.radix.warpHist[warp][d] = __popc( peers );
			__syncthreads();
			unsigned run = 0;
			if ( tid < 256 )
			{
				for ( int w = 0; w < CSORT_WARPS; ++w )
				{
					unsigned t = sm.radix.warpHist[w][tid];
					sm.radix.warpHist[w][tid] = run;
					run += t;
				}
			}
			__syncthreads();
			if ( valid )
			{
				unsigned dst = sm.radix.base[d] + sm.radix.warpHist[warp][d] + rank;
				kout[dst] = key;
				if ( vout )
					vout[dst] = val;
			}
			__syncthreads();
			if ( tid < 256 )
				sm.radix.base[tid] += run;
			__syncthreads();
		}
		if ( !grid_barrier( counter, err, epoch ) )
			return;
		K* tk = kin;
		kin = kout;
		kout = tk;
		int* tv = vin;
		vin = vout;
		vout = tv;
	}
	if ( done & 1 )
	{
		// the rows ended in the alternate buffers: copy this block's range back
		for ( int i = lo + tid; i < hi; i += CSORT_THREADS )
		{
			keys[i] = __ldcg( kin + i );
			if ( vals )
				vals[i] = __ldcg( vin + i );
		}
	}
	if ( dec.made )
		for ( int i = lo + tid; i < hi; i += CSORT_THREADS )
			dec.made[i] = dec.lookup[__ldcg( kin + i ) >> dec.shift];
}

// Sorts (keys, vals) by the low `bits` bits of the keys; vals may be null.
// n from device memory, at most cap rows are sorted. `large`: a world whose
// sorts commonly pass CSORT_SMALL rows (SORT_LARGE_WORLD) launches the
// one-block sort ahead of the cooperative one; in a smaller world that launch
// would be 2.3 us of nothing in every step. hist needs 256 * CSORT_MAX_BLOCKS unsigned; counter
// is a device word used by the grid barrier (zero before the launch, one
// launch per step and word). When enable is
// non-null the sort runs only if *enable != 0.
template <typename K>
static inline void sort_coop( K* keys, int* vals, K* keysAlt, int* valsAlt, int* nPtr, int cap, int bits,
							  unsigned* hist, unsigned* counter, int* err, int blocks, cudaStream_t st,
							  const int* enable, bool large, SortDecode dec = { nullptr, nullptr, 0 } )
{
	if ( blocks > CSORT_MAX_BLOCKS )
		blocks = CSORT_MAX_BLOCKS;
	if ( vals == nullptr )
		valsAlt = nullptr;
	int skipUpTo = 0;
	if ( large )
	{
		cudaFuncSetAttribute( k_sort_block<K>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof( BSortSmem ) );
		k_sort_block<K><<<1, CSORT_THREADS, sizeof( BSortSmem ), st>>>( keys, vals, nPtr, cap, bits, enable, dec );
		skipUpTo = BSORT_MAX;
	}
	void* args[] = { &keys, &vals, &keysAlt, &valsAlt, &nPtr, &cap, &bits, &hist, &counter, &err, &enable, &skipUpTo, &dec };
	cudaLaunchCooperativeKernel( (void*)k_sort_coop<K>, dim3( blocks ), dim3( CSORT_THREADS ), args, 0, st );
}

// Co-resident block count for k_sort_coop on the current device.
template <typename K> static inline int sort_coop_blocks()
{
	int perSM = 0;
	cudaOccupancyMaxActiveBlocksPerMultiprocessor( &perSM, k_sort_coop<K>, CSORT_THREADS, 0 );
	int dev = 0, sms = 0;
	cudaGetDevice( &dev );
	cudaDeviceGetAttribute( &sms, cudaDevAttrMultiProcessorCount, dev );
	int b = perSM >= 1 ? sms : 0;
	return b > CSORT_MAX_BLOCKS ? CSORT_MAX_BLOCKS : b;
}

// Compaction in one launch: blocks of LOOKBACK_TILE threads, an item each, tiles
// chained by decoupled look-back (state zeroed before the launch, one launch
// per step and state). Calls place( item, slot ) for the wanted items, slots in
// item order, and finish( count ) once.
template <typename Want, typename Place, typename Finish>
__device__ __forceinline__ void compact_items( unsigned long long* state, int n, int* err, Want want, Place place, Finish finish )
{
	__shared__ int smem[32];
	__shared__ int s_tile, s_prefix;
	if ( threadIdx.x == 0 )
		s_tile = (int)atomicAdd( (unsigned*)state, 1u );
	__syncthreads();
	const int tile = s_tile, base = tile * LOOKBACK_TILE;
	if ( base >= n )
	{
		if ( tile == 0 && threadIdx.x == 0 )
			finish( 0 );
		return;
	}
	const int item = base + threadIdx.x;
	const bool wanted = item < n && want( item );
	int total;
	const int slot = block_exclusive_scan_1024( wanted ? 1 : 0, smem, &total );
	if ( threadIdx.x < 32 )
	{
		if ( threadIdx.x == 0 )
			lookback_publish( state + 1, tile, total );
		__syncwarp();
		const int prefix = lookback_prefix( state + 1, tile, total, err );
		if ( threadIdx.x == 0 )
		{
			s_prefix = prefix;
			if ( base + LOOKBACK_TILE >= n )
				finish( prefix + total );
		}
	}
	__syncthreads();
	if ( wanted )
		place( item, s_prefix + slot );
}

static inline int compact_blocks( int cap )
{
	return ( cap + LOOKBACK_TILE - 1 ) / LOOKBACK_TILE;
}

// ---------------------------------------------------------------------------
// exclusive scan with decoupled look-back
// state[0]: tile ticket; state[1 + t]: tile t's flag (bits 32..33) and value
// ---------------------------------------------------------------------------
static __global__ void __launch_bounds__( LB_THREADS )
	k_scan_lookback( const int* __restrict__ in, int* __restrict__ out, const int* __restrict__ nPtr, int nConst,
					 unsigned long long* state, int* __restrict__ totalOut, int* err, const int* enable )
{
	__shared__ int smem[32];
	__shared__ int s_tile, s_prefix;
	if ( enable && *enable == 0 )
		return;
	int n = nPtr ? *nPtr : nConst;
	if ( threadIdx.x == 0 )
		s_tile = (int)atomicAdd( (unsigned*)state, 1u );
	__syncthreads();
	int tile = s_tile;
	int base = tile * LB_TILE;
	if ( base >= n )
	{
		if ( tile == 0 && threadIdx.x == 0 && totalOut )
			*totalOut = 0;
		return;
	}
	int v[LB_ITEMS];
	int sum = 0;
#pragma unroll
	for ( int k = 0; k < LB_ITEMS; ++k )
	{
		int i = base + threadIdx.x * LB_ITEMS + k;
		v[k] = i < n ? in[i] : 0;
		sum += v[k];
	}
	int aggregate;
	int excl = block_exclusive_scan_1024( sum, smem, &aggregate );
	if ( threadIdx.x == 0 )
	{
		int prefix = 0;
		if ( tile == 0 )
			st_release_u64( state + 1, ( LB_FLAG_PREFIX << 32 ) | (unsigned)aggregate );
		else
		{
			st_release_u64( state + 1 + tile, ( LB_FLAG_AGG << 32 ) | (unsigned)aggregate );
			int j = tile - 1;
			long long spins = 0;
			while ( j >= 0 )
			{
				unsigned long long s = ld_acquire_u64( state + 1 + j );
				unsigned long long flag = s >> 32;
				if ( flag == 0ull )
				{
					if ( ++spins > F2D_SPIN_LIMIT )
					{
						atomicOr( err, F2D_ERR_BARRIER_TIMEOUT );
						break;
					}
					continue;
				}
				prefix += (int)(unsigned)( s & 0xffffffffull );
				if ( flag == LB_FLAG_PREFIX )
					break;
				j -= 1;
			}
			st_release_u64( state + 1 + tile, ( LB_FLAG_PREFIX << 32 ) | (unsigned)( prefix + aggregate ) );
		}
		s_prefix = prefix;
		if ( totalOut && base + LB_TILE >= n )
			*totalOut = prefix + aggregate;
	}
	__syncthreads();
	excl += s_prefix;
#pragma unroll
	for ( int k = 0; k < LB_ITEMS; ++k )
	{
		int i = base + threadIdx.x * LB_ITEMS + k;
		if ( i < n )
			out[i] = excl;
		excl += v[k];
	}
}

// Exclusive scan of n ints (n from nPtr when non-null, else nConst); cap
// bounds the grid; state needs cap / LB_TILE + 2 words; totalOut (device)
// receives the sum when non-null. When enable is non-null the scan runs only
// if *enable != 0.
static inline void scan_lookback( const int* in, int* out, const int* nPtr, int nConst, int cap, int* totalOut,
								  unsigned long long* state, int* err, cudaStream_t st,
								  const int* enable = nullptr )
{
	int tiles = ( cap + LB_TILE - 1 ) / LB_TILE;
	if ( tiles < 1 )
		tiles = 1;
	cudaMemsetAsync( state, 0, sizeof( unsigned long long ) * (size_t)( tiles + 1 ), st );
	k_scan_lookback<<<tiles, LB_THREADS, 0, st>>>( in, out, nPtr, nConst, state, totalOut, err, enable );
}
