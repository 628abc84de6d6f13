// Device exclusive prefix sum of uint32 counts (tile activation flags, per-dual-cell
// particle counts). Up to 8192 counts: one block. Up to 16 M: per-block sums (2048 elements per
// block), then a scan per block whose offset the block sums up itself from the block sums before
// it, its elements read ahead of the wait for them. Beyond, where those sums would be most of the
// traffic: a one-block scan of the block sums in between. Each pass reads its input with 128-bit
// loads; the block-sum scratch array is owned by the caller. Latency bounds the small ones: 11.3 us
// with three launches up to 100 K counts, 4.2 in one block (8192), 6.1 with two launches; 20.5 and
// 12.3 us for 4 M.
#include "bora_internal.h"

namespace {

constexpr int kScanThreads = 256;
constexpr int kScanItems = 8;  // per thread -> 2048 elements per block
constexpr int kScanChunk = kScanThreads * kScanItems;
constexpr int kScanOneThreads = 1024;
constexpr size_t kScanOneMax = (size_t)kScanOneThreads * kScanItems;
constexpr int kScanSelfMax = 8192;  // blocks up to which a block sums up its own offset (16 M counts: 41.0 us, 53.3 with three launches)

__device__ inline uint32_t warp_incl_scan( uint32_t v )
{
    const int lane = threadIdx.x & 31;
#pragma unroll
    for( int o = 1; o < 32; o <<= 1 )
    {
        const uint32_t t = __shfl_up_sync( 0xffffffffu, v, o );
        if( lane >= o ) v += t;
    }
    return v;
}

// Block-wide exclusive scan of one value per thread; returns the exclusive prefix and
// the block total in *total.
template <int T>
__device__ inline uint32_t block_excl_scan( uint32_t v, uint32_t* total )
{
    __shared__ uint32_t warp_sums[T / 32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const uint32_t inc = warp_incl_scan( v );
    if( lane == 31 ) warp_sums[wid] = inc;
    __syncthreads();
    if( wid == 0 )
    {
        uint32_t s = lane < T / 32 ? warp_sums[lane] : 0u;
        s = warp_incl_scan( s );
        if( lane < T / 32 ) warp_sums[lane] = s;
    }
    __syncthreads();
    const uint32_t base = wid > 0 ? warp_sums[wid - 1] : 0u;
    *total = warp_sums[T / 32 - 1];
    __syncthreads();
    return base + inc - v;
}

__device__ inline void load_items( const uint32_t* __restrict__ in, size_t n, size_t base, uint32_t v[kScanItems] )
{
    const size_t i0 = base + (size_t)threadIdx.x * kScanItems;
    if( i0 + kScanItems <= n && ( ( reinterpret_cast<uintptr_t>( in + i0 ) & 15 ) == 0 ) )
    {
        const uint4 a = *reinterpret_cast<const uint4*>( in + i0 );
        const uint4 b = *reinterpret_cast<const uint4*>( in + i0 + 4 );
        v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
        v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
    }
    else
    {
#pragma unroll
        for( int q = 0; q < kScanItems; ++q ) v[q] = ( i0 + q < n ) ? in[i0 + q] : 0u;
    }
}

__device__ inline uint32_t item_sum( const uint32_t v[kScanItems] )
{
    uint32_t s = 0;
#pragma unroll
    for( int q = 0; q < kScanItems; ++q ) s += v[q];
    return s;
}

// the thread's items as prefix sums from `run`
__device__ inline void store_items( uint32_t* __restrict__ out, size_t n, size_t base, const uint32_t v[kScanItems], uint32_t run )
{
    const size_t i0 = base + (size_t)threadIdx.x * kScanItems;
    uint32_t o[kScanItems];
#pragma unroll
    for( int q = 0; q < kScanItems; ++q ) { o[q] = run; run += v[q]; }
    if( i0 + kScanItems <= n && ( ( reinterpret_cast<uintptr_t>( out + i0 ) & 15 ) == 0 ) )
    {
        *reinterpret_cast<uint4*>( out + i0 ) = make_uint4( o[0], o[1], o[2], o[3] );
        *reinterpret_cast<uint4*>( out + i0 + 4 ) = make_uint4( o[4], o[5], o[6], o[7] );
    }
    else
    {
#pragma unroll
        for( int q = 0; q < kScanItems; ++q )
            if( i0 + q < n ) out[i0 + q] = o[q];
    }
}

// n <= kScanOneMax
__global__ void __launch_bounds__( kScanOneThreads ) k_scan_one( const uint32_t* in, size_t n, uint32_t* out,
                                                                 uint32_t* __restrict__ grand_total )
{
    uint32_t v[kScanItems];
    load_items( in, n, 0, v );
    uint32_t total;
    const uint32_t run = block_excl_scan<kScanOneThreads>( item_sum( v ), &total );
    store_items( out, n, 0, v, run );
    if( threadIdx.x == 0 && grand_total ) *grand_total = total;
}

__global__ void k_scan_reduce( const uint32_t* __restrict__ in, size_t n, uint32_t* __restrict__ block_sums )
{
    bora_pdl_trigger();
    uint32_t v[kScanItems];
    load_items( in, n, (size_t)blockIdx.x * kScanChunk, v );
    uint32_t total;
    block_excl_scan<kScanThreads>( item_sum( v ), &total );
    if( threadIdx.x == 0 ) block_sums[blockIdx.x] = total;
}

// One block scans the nb block sums in place (exclusive) and writes the grand total.
__global__ void k_scan_blocks( uint32_t* __restrict__ block_sums, int nb, uint32_t* __restrict__ grand_total )
{
    uint32_t carry = 0;
    for( int base = 0; base < nb; base += kScanThreads )
    {
        const int i = base + threadIdx.x;
        const uint32_t v = i < nb ? block_sums[i] : 0u;
        uint32_t total;
        const uint32_t ex = block_excl_scan<kScanThreads>( v, &total );
        if( i < nb ) block_sums[i] = carry + ex;
        carry += total;
    }
    if( threadIdx.x == 0 && grand_total ) *grand_total = carry;
}

// SELF: block_sums are the blocks' sums (the kernel follows k_scan_reduce, which no longer reads
// `in` when a block of this one writes); else they are scanned already.
template <bool SELF>
__global__ void __launch_bounds__( kScanThreads ) k_scan_down( const uint32_t* in, size_t n, const uint32_t* block_sums,
                                                               uint32_t* out, uint32_t* __restrict__ grand_total )
{
    uint32_t v[kScanItems];
    const size_t base = (size_t)blockIdx.x * kScanChunk;
    load_items( in, n, base, v );
    uint32_t total, offset = 0;
    uint32_t run = block_excl_scan<kScanThreads>( item_sum( v ), &total );
    if( SELF )
    {
        bora_pdl_wait();
        uint32_t before = 0;
        for( unsigned b = threadIdx.x; b < blockIdx.x; b += kScanThreads ) before += block_sums[b];
        block_excl_scan<kScanThreads>( before, &offset );
        if( grand_total && blockIdx.x == gridDim.x - 1 && threadIdx.x == 0 ) *grand_total = offset + total;
    }
    else offset = block_sums[blockIdx.x];
    store_items( out, n, base, v, run + offset );
}

}  // namespace

size_t bora_scan_scratch_elems( size_t n ) { return ( n + kScanChunk - 1 ) / kScanChunk + 1; }

// out[i] = sum_{j<i} in[i]; *total = sum of all (device pointer, may be null).
// in and out may alias. scratch holds bora_scan_scratch_elems(n) uint32.
// Returns its kernel launches.
int bora_device_scan( const uint32_t* in, uint32_t* out, size_t n, uint32_t* scratch, uint32_t* total, cudaStream_t st )
{
    if( n == 0 )
    {
        if( total ) cudaMemsetAsync( total, 0, sizeof( uint32_t ), st );
        return 0;
    }
    if( n <= kScanOneMax )
    {
        k_scan_one<<<1, kScanOneThreads, 0, st>>>( in, n, out, total );
        return 1;
    }
    const int nb = (int)( ( n + kScanChunk - 1 ) / kScanChunk );
    k_scan_reduce<<<nb, kScanThreads, 0, st>>>( in, n, scratch );
    if( nb <= kScanSelfMax )
    {
        bora_launch_pdl( k_scan_down<true>, dim3( nb ), dim3( kScanThreads ), 0, st, in, n, (const uint32_t*)scratch, out, total );
        return 2;
    }
    k_scan_blocks<<<1, kScanThreads, 0, st>>>( scratch, nb, total );
    k_scan_down<false><<<nb, kScanThreads, 0, st>>>( in, n, scratch, out, nullptr );
    return 3;
}

// ---- public C ABI: device exclusive prefix sum -------------------------------------
#include "../../include/bora_flip.h"

extern "C" int bora_scan_u32( const uint32_t* d_in, uint32_t* d_out, size_t n, uint32_t* d_total, void* stream )
{
    if( n > 0 && ( !d_in || !d_out ) ) return BORA_ERR_INVALID_ARG;
    if( n > (size_t)0xFFFFFFFFu ) return BORA_ERR_CAPACITY;
    cudaStream_t st = (cudaStream_t)stream;
    uint32_t* scratch = nullptr;
    if( n > 0 )
    {
        // stream-ordered scratch for the per-block sums, released on the same stream
        const cudaError_t e = cudaMallocAsync( (void**)&scratch, bora_scan_scratch_elems( n ) * sizeof( uint32_t ), st );
        if( e != cudaSuccess ) return e == cudaErrorMemoryAllocation ? BORA_ERR_OUT_OF_MEMORY : BORA_ERR_CUDA;
    }
    bora_device_scan( d_in, d_out, n, scratch, d_total, st );
    cudaError_t e = cudaGetLastError();
    if( scratch )
    {
        const cudaError_t f = cudaFreeAsync( scratch, st );
        if( e == cudaSuccess ) e = f;
    }
    return e == cudaSuccess ? BORA_OK : BORA_ERR_CUDA;
}

// ---- no-allocation variant ---------------------------------------------------------
// For callers that must not allocate device memory (see bora_scan_u32_noalloc in
// include/bora_flip.h). The per-block sums live in this file-scope array: 2048 input
// counts per block, so 2^28 counts need 131,073 sums (512 KiB + 4 B). Every device that
// loads the library holds the array until the process exits.
#include <mutex>

#define BORA_SCAN_NOALLOC_MAX ( (size_t)1 << 28 )
static __device__ __align__( 256 ) uint32_t g_noalloc_block_sums[BORA_SCAN_NOALLOC_MAX / kScanChunk + 1];

namespace {
std::mutex g_noalloc_mutex;
uint32_t* g_noalloc_addr[64] = {};  // device address of g_noalloc_block_sums, per device ordinal
}  // namespace

extern "C" int bora_scan_u32_noalloc( const uint32_t* d_in, uint32_t* d_out, size_t n, uint32_t* d_total, void* stream )
{
    if( n > 0 && ( !d_in || !d_out ) ) return BORA_ERR_INVALID_ARG;
    if( n > BORA_SCAN_NOALLOC_MAX ) return BORA_ERR_CAPACITY;
    int dev = -1;
    if( cudaGetDevice( &dev ) != cudaSuccess || dev < 0 || dev >= 64 ) return BORA_ERR_CUDA;
    uint32_t* scratch = nullptr;
    {
        // First call on this device: the host-side name of the array is not a device
        // address, so ask the runtime for the address on the current device.
        std::lock_guard<std::mutex> lock( g_noalloc_mutex );
        if( !g_noalloc_addr[dev] )
        {
            void* p = nullptr;
            if( cudaGetSymbolAddress( &p, g_noalloc_block_sums ) != cudaSuccess || !p ) return BORA_ERR_CUDA;
            g_noalloc_addr[dev] = static_cast<uint32_t*>( p );
        }
        scratch = g_noalloc_addr[dev];
    }
    // Each call writes every block sum before reading it, so the array's previous
    // contents never matter and nothing needs clearing.
    bora_device_scan( d_in, d_out, n, scratch, d_total, (cudaStream_t)stream );
    return cudaGetLastError() == cudaSuccess ? BORA_OK : BORA_ERR_CUDA;
}
