// FP64-accurate, deterministic reductions shared by the solver kernels.
#pragma once

#include <cstring>

#include "bora_internal.h"

namespace bora_reduce {

// ---------------------------------------------------------------------------------
// Double-float accumulation: GB300's FP64 pipe is ~1/64 of its FP32 rate, so per-cell
// dot-product terms are accumulated as unevaluated float pairs (hi + lo) with the
// error-free TwoProd (fmaf) and TwoSum transformations (Dekker 1971, Knuth TAOCP 4.2.2),
// giving ~48 significant bits from FP32 instructions; each warp converts its pair to
// FP64 once. The product is formed with __fmul_rn, which the compiler never fuses into a
// following addition, so the transformations stay error-free under -fmad=true as well
// (TwoSum has no multiplication to contract).
struct DF
{
    float hi, lo;
};
__device__ __forceinline__ DF df_prod( float a, float b )
{
    const float p = __fmul_rn( a, b );
    return DF{ p, fmaf( a, b, -p ) };
}
__host__ __device__ __forceinline__ DF df_add( DF a, DF b )
{
    const float s = a.hi + b.hi;
    const float bb = s - a.hi;
    float err = ( a.hi - ( s - bb ) ) + ( b.hi - bb );
    err += a.lo + b.lo;
    const float h = s + err;
    return DF{ h, err - ( h - s ) };
}
// DF + float (TwoSum with a zero low part).
__device__ __forceinline__ DF df_add_f( DF a, float b )
{
    const float s = a.hi + b;
    const float bb = s - a.hi;
    const float err = ( ( a.hi - ( s - bb ) ) + ( b - bb ) ) + a.lo;
    const float h = s + err;
    return DF{ h, err - ( h - s ) };
}
// FP32 dot product of two float4 (fused multiply-adds). Short FP32 partial sums like this
// one (4 terms, relative error ~2^-22) feed the double-float accumulators: that keeps the
// totals accurate to ~1e-7 relative, far more than the FP32 alpha and beta of PCG need,
// at a quarter of the double-float operations.
__device__ __forceinline__ float dot4( float4 a, float4 b )
{
    return fmaf( a.w, b.w, fmaf( a.z, b.z, fmaf( a.y, b.y, a.x * b.x ) ) );
}
__device__ __forceinline__ double df_warp_sum( DF v )
{
#pragma unroll
    for( int o = 16; o > 0; o >>= 1 )
    {
        DF w;
        w.hi = __shfl_xor_sync( 0xffffffffu, v.hi, o );
        w.lo = __shfl_xor_sync( 0xffffffffu, v.lo, o );
        v = df_add( v, w );
    }
    return (double)v.hi + (double)v.lo;
}
__device__ __forceinline__ float warp_maxf( float v )
{
#pragma unroll
    for( int o = 16; o > 0; o >>= 1 ) v = fmaxf( v, __shfl_xor_sync( 0xffffffffu, v, o ) );
    return v;
}

// ---------------------------------------------------------------------------------
// Deterministic FP64 block reduction published through a ring slot: every block writes
// its partial, the last block to arrive sums the partials in block order.
__device__ __forceinline__ double warp_sum( double v )
{
#pragma unroll
    for( int o = 16; o > 0; o >>= 1 ) v += __shfl_xor_sync( 0xffffffffu, v, o );
    return v;
}
__device__ __forceinline__ double warp_max( double v )
{
#pragma unroll
    for( int o = 16; o > 0; o >>= 1 ) v = fmax( v, __shfl_xor_sync( 0xffffffffu, v, o ) );
    return v;
}

// A sum (v0) and a maximum (v1), the per-warp totals (already reduced across the warp, valid in
// every lane). The block takes part as block `bid` of `nblocks` (blockIdx.x of gridDim.x unless a
// batched launch runs several simulations' blocks side by side).
__device__ __forceinline__ void reduce2_publish_warp( double v0, double v1, BoraReduceDev red, int slot0, int slot1, unsigned bid,
                                                      unsigned nblocks )
{
    __shared__ double w0[32], w1[32];
    __shared__ bool last;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = ( blockDim.x + 31 ) >> 5;
    if( lane == 0 ) { w0[wid] = v0; w1[wid] = v1; }
    __syncthreads();
    if( threadIdx.x == 0 )
    {
        double a = 0.0, b = 0.0;
        for( int q = 0; q < nw; ++q ) { a += w0[q]; b = fmax( b, w1[q] ); }
        red.partials[2 * (size_t)bid] = a;
        red.partials[2 * (size_t)bid + 1] = b;
        __threadfence();
        const unsigned prev = atomicAdd( &red.done[slot0 % BORA_RING], 1u );
        last = ( prev == nblocks - 1 );
    }
    __syncthreads();
    if( !last ) return;
    __threadfence();
    // All threads of the last block: thread-strided partial sums in a fixed order
    // (independent loads, unrolled so that many are in flight), then a fixed-shape tree.
    double a = 0.0, b = 0.0;
    const unsigned nb = nblocks, stride = blockDim.x;
#pragma unroll 4
    for( unsigned q = threadIdx.x; q < nb; q += stride )
    {
        const double2 pq = __ldcg( reinterpret_cast<const double2*>( red.partials ) + q );
        a += pq.x;
        b = fmax( b, pq.y );
    }
    a = warp_sum( a );
    b = warp_max( b );
    if( lane == 0 ) { w0[wid] = a; w1[wid] = b; }
    __syncthreads();
    if( threadIdx.x == 0 )
    {
        double ta = 0.0, tb = 0.0;
        for( int q = 0; q < nw; ++q ) { ta += w0[q]; tb = fmax( tb, w1[q] ); }
        red.ring[slot0] = ta;
        const float hi = (float)ta;
        red.ringf[slot0] = make_float2( hi, (float)( ta - (double)hi ) );
        red.ring[slot1] = tb;
        if( red.mirror )  // the host polls them
        {
            red.mirror[slot0] = ta;
            red.mirror[slot1] = tb;
        }
        red.done[slot0 % BORA_RING] = 0;
        __threadfence();
    }
}

// Per-thread double-float sums and float maxima.
__device__ __forceinline__ void reduce2_publish_dfmax( DF v0, float vmax, BoraReduceDev red, int slot0, int slot1,
                                                       unsigned bid, unsigned nblocks )
{
    const double a = df_warp_sum( v0 );
    const double b = (double)warp_maxf( vmax );
    reduce2_publish_warp( a, b, red, slot0, slot1, bid, nblocks );
}


// ---------------------------------------------------------------------------------
// Sums finished by their consumer. The solver's inner kernels run as a chain in which the next
// kernel needs the previous one's sum: a producer's block stores its partial sum as a
// double-float pair and exits, and every block of the consumer adds all partials in the same
// fixed order while its first tile's loads are in flight, so each holds the same bits. Against
// a last block that finishes the sum (fence, arrival counter, second pass, 7 us at the end of
// every reducing kernel on GB300: 13.8 against 6.4 us for level 0's down passes with and
// without a sum at 240 tiles), the producer's tail is one store. Partials are float pairs
// (48 bits): FP64 additions by every block would be bound by the narrow FP64 pipe. Measured
// with the host polling r.r instead of waiting for events: a plain PCG iteration at 240 tiles
// 18 -> 13 us, the 256^3 plain step's solve 32 -> 27 ms, a V-cycle 6 us less.

__device__ __forceinline__ DF df_warp_sum_df( DF v )
{
#pragma unroll
    for( int o = 16; o > 0; o >>= 1 )
        v = df_add( v, DF{ __shfl_xor_sync( 0xffffffffu, v.hi, o ), __shfl_xor_sync( 0xffffffffu, v.lo, o ) } );
    return v;
}

// (float)( a / b ) of two double-float values: the quotient of the high parts corrected by one
// residual step, which rounds the quotient of the pairs once (off by 0.5 + 2^-22 ulp at most, as
// the FP64 quotient rounded to FP32). Small operands are scaled by a power of two, so that the
// remainder does not lose bits below FP32's smallest normal number.
__host__ __device__ __forceinline__ float df_ratio( float2 a, float2 b )
{
    constexpr float kSmall = 1e-20f, kUp = 1.152921504606847e18f, kDown = 1.f / kUp;  // 2^60
    float back = 1.f;
    if( fabsf( a.x ) < kSmall ) { a.x *= kUp; a.y *= kUp; back = kDown; }
    if( fabsf( b.x ) < kSmall ) { b.x *= kUp; b.y *= kUp; back *= kUp; }
    const float q = a.x / b.x;
    const float rem = fmaf( -q, b.x, a.x ) + fmaf( -q, b.y, a.y );
    const float c = rem / b.x;
    return ( isfinite( c ) ? q + c : q ) * back;
}

// The V-cycle's scale of a residual with r.r = rr: the power of two 2^-k with 2^k <= sqrt( rr ) < 2^(k + 1),
// within FP32's normal range (1 for rr = 0 or not finite). A product with it, and with its
// reciprocal, is exact; a quotient by the norm's root would be rounded twice per cell.
__host__ __device__ __forceinline__ float residual_scale( double rr )
{
    unsigned long long u;
    memcpy( &u, &rr, 8 );
    if( !( rr > 0.0 ) || u >> 52 == 0x7ffu ) return 1.f;
    const int k = ( (int)( u >> 52 ) - 1023 ) >> 1;  // from the exponents' bits: 2^(2k) <= rr < 2^(2k + 2)
    const unsigned w = (unsigned)( 127 - ( k < -126 ? -126 : ( k > 126 ? 126 : k ) ) ) << 23;
    float sc;
    memcpy( &sc, &w, 4 );
    return sc;
}

// The block's sums of v0 and v1 into part0[bid] and part1[bid] (part1 may be null). Called once per
// kernel, by every thread of the block.
__device__ __forceinline__ void part_publish( DF v0, DF v1, float2* part0, float2* part1, unsigned bid )
{
    __shared__ float4 w[32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = ( blockDim.x + 31 ) >> 5;
    v0 = df_warp_sum_df( v0 );
    if( part1 ) v1 = df_warp_sum_df( v1 );
    if( lane == 0 ) w[wid] = make_float4( v0.hi, v0.lo, v1.hi, v1.lo );
    __syncthreads();
    if( threadIdx.x == 0 )
    {
        DF a{ w[0].x, w[0].y }, b{ w[0].z, w[0].w };
        for( int q = 1; q < nw; ++q )
        {
            a = df_add( a, DF{ w[q].x, w[q].y } );
            b = df_add( b, DF{ w[q].z, w[q].w } );
        }
        part0[bid] = make_float2( a.hi, a.lo );
        if( part1 ) part1[bid] = make_float2( b.hi, b.lo );
    }
}

// The sum of part[0 .. n) in a fixed order that depends on n and the block's size alone, returned in
// every thread. Every thread of the block calls it; w is shared memory of the caller, one
// float2 per warp, not used by anything else since the last block barrier.
__device__ __forceinline__ DF part_collect( const float2* part, int n, float2* w )
{
    constexpr int kAhead = 8;  // independent loads in flight per thread
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = ( blockDim.x + 31 ) >> 5;
    DF a{ 0.f, 0.f };
    for( int base = threadIdx.x; base < n; base += kAhead * (int)blockDim.x )
    {
        float2 p[kAhead];
#pragma unroll
        for( int q = 0; q < kAhead; ++q )
        {
            const int i = base + q * (int)blockDim.x;
            p[q] = i < n ? __ldcg( part + i ) : make_float2( 0.f, 0.f );
        }
#pragma unroll
        for( int q = 0; q < kAhead; ++q ) a = df_add( a, DF{ p[q].x, p[q].y } );
    }
    a = df_warp_sum_df( a );
    if( lane == 0 ) w[wid] = make_float2( a.hi, a.lo );
    __syncthreads();
    DF t{ w[0].x, w[0].y };
    for( int q = 1; q < nw; ++q ) t = df_add( t, DF{ w[q].x, w[q].y } );
    return t;
}

// A finished sum for the kernels after this one, and (mirror) for the host. One thread calls it.
__device__ __forceinline__ void ring_store( const BoraReduceDev& red, int slot, DF v, bool mirror )
{
    red.ringf[slot] = make_float2( v.hi, v.lo );
    red.ring[slot] = (double)v.hi + (double)v.lo;
    if( mirror && red.mirror ) red.mirror[slot] = (double)v.hi + (double)v.lo;
}

}  // namespace bora_reduce

using namespace bora_reduce;
