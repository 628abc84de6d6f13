// The tiled levels of the multigrid V-cycle (levels 0, 1, 2: 8^3, 4^3 and 2^3 cells per
// tile) as stencil passes over each level's own cells.
//
// A level is pre-smoothed and restricted in two passes and prolonged and post-smoothed in
// two more; every pass is a 7-point stencil that reads its neighbours' values of one field:
//   down 1  z2 = S_B(S_A(0)). The first sweep from zero is pointwise, z1 = w_A r' / d, so
//           the second reads its neighbours' r' and codes.                      z2 -> scratch
//   down 2  res = r' - A z2 (the neighbours' z2); z0 = FP16(z2); the coarser level's
//           r = FP16(0.5 * sum of the 8 children's res)
//   up 1    za = z0 + e(parent) (injection of the coarser correction), zb = S_B(za) (the
//           neighbours' za).                                                    zb -> scratch
//   up 2    z = S_A(zb) (the neighbours' zb); level 0 unscales into the FP32 z of the PCG and
//           sums r.z, the other levels store FP16 z1 for the finer level's up 1
// where r' = r * sc on level 0 (sc = the power of two that brings ||r|| of the latest residual whose
// norm is known to [1, 2): it keeps the FP16 levels' values O(1), scaling and unscaling are exact,
// and the V-cycle is linear in r, so any scale serves) and r on the others,
// S_w(v) = v + (w / d) (r' - (d v - sum of the neighbours' v)) on fluid cells and 0 elsewhere,
// neighbour sums in the order ((x- + x+) + (y- + y+)) + (z- + z+), and the 8 children summed as
// ((x pairs) + (y pairs)) + (z pairs). Every cell is computed once per pass; the scratch is
// the FP32 cell vector that the plain form keeps its preconditioner pivots in (the mixed form
// has none), used by one pass pair at a time: level 0 stores its z2 and zb there in FP16 (half
// the bytes of the pass pair's store and reads; the residual of down 2 is then formed from the
// same FP16 values that z0 keeps), levels 1 and 2 in FP32.
//
// Level 0's down passes also apply the PCG's residual update r -= alpha q (alpha = rz / dq of the
// last direction): down 1 forms the updated residual of its cells and of the face cells it reads,
// without storing it, and sums r.r over the grid (the convergence check); down 2, which reads no
// neighbour's r, stores it. This takes the update kernel out of every iteration.
//
// Level 0 runs one warp per half tile (z layers 0..3 or 4..7): a lane owns one x-row (lane =
// j + 8 (k mod 4)), read and written as whole vectors; its x neighbours are in its registers, the
// y and z neighbours come from other lanes by shuffles, and the lanes at the half's faces load
// the rows across them (the other half, the neighbour tiles). The passes wait on their loads, so
// they want warps in flight and all of a lane's loads issued before the first is used: with a
// tile per warp (two rows per lane, 128 registers, 12 warps in flight) the four passes took 33,
// 18, 28 and 24 us at 256^3 (8.2 K tiles). Levels 1 and 2 run one
// thread per x-row of 4 or 2 cells.
#include <algorithm>
#include <type_traits>

#include "bora_internal.h"
#include "reduce.cuh"

namespace {

constexpr float kOmegaA = 0.5687f;  // the Chebyshev pair of the smoothers (multigrid.cu)
constexpr float kOmegaB = 1.6902f;
// launch shapes (the autotuner picks one per size class; the results do not depend on it):
// level 0 half tiles (warps) per block, levels 1 and 2 threads (x-rows) per block
constexpr int kPassWarpsOf[3] = { 2, 4, 8 };
constexpr int kFlatThreadsOf[4] = { 64, 128, 256, 512 };
// Warps per SM that level 0 asks registers for: 24 (80 registers) for down 2 and up 1, 16 (128)
// for the reducing passes (down 1 holds code, r and q of two halo rows). A 256^3 mixed step
// takes 4.08 ms with 24 / 16, 4.13 with 24 / 20, 4.14 with 24 / 24 (down 1 spills), 4.11 with
// 16 / 16, 4.15 with 32 / 20 (spills); 4.54 with a whole tile per warp at 128 registers.
constexpr int kPassWarpsPerSm = 24, kReduceWarpsPerSm = 16;
constexpr int pass_warps_per_sm( int P ) { return P == 0 || P == 3 ? kReduceWarpsPerSm : kPassWarpsPerSm; }
constexpr int kReduceWarps = 4;  // level 0's up 2 sums r.z over its blocks: its shape is fixed
constexpr unsigned kAll = 0xffffffffu;

__device__ __forceinline__ int cdiag( uint16_t c ) { return ( c >> 8 ) & 15; }
__device__ __forceinline__ bool cfluid( uint16_t c ) { return ( c & BORA_CODE_FLUID ) != 0; }

// w / d for d = 0..15 (0 for d = 0): w_A in [0, 16), w_B in [16, 32)
__device__ __forceinline__ void init_weights( float* w )
{
    const int t = threadIdx.x;
    if( t < 32 )
    {
        const int d = t & 15;
        w[t] = d ? ( t < 16 ? kOmegaA : kOmegaB ) / (float)d : 0.f;
    }
}

// one damped Jacobi update of cell value v from its neighbour sum (w = w_A or w_B table)
__device__ __forceinline__ float sweep( float v, float r, uint16_t c, float sum, const float* w )
{
    return cfluid( c ) ? v + w[cdiag( c )] * ( r - ( (float)cdiag( c ) * v - sum ) ) : 0.f;
}

// ---- level 0: one warp per half tile ---------------------------------------------------------

__device__ __forceinline__ void codes8( uint4 w, uint16_t* c )
{
    const uint32_t a[4] = { w.x, w.y, w.z, w.w };
#pragma unroll
    for( int i = 0; i < 4; ++i )
    {
        c[2 * i] = (uint16_t)( a[i] & 0xffffu );
        c[2 * i + 1] = (uint16_t)( a[i] >> 16 );
    }
}

__device__ __forceinline__ float hbits( uint32_t w, int q ) { return __half2float( __ushort_as_half( (unsigned short)( w >> ( 16 * q ) ) ) ); }

__device__ __forceinline__ void f16x8( uint4 w, float* v )
{
    const uint32_t a[4] = { w.x, w.y, w.z, w.w };
#pragma unroll
    for( int i = 0; i < 4; ++i ) { v[2 * i] = hbits( a[i], 0 ); v[2 * i + 1] = hbits( a[i], 1 ); }
}

__device__ __forceinline__ uint32_t pack2( float a, float b )
{
    return (uint32_t)__half_as_ushort( __float2half_rn( a ) ) | ( (uint32_t)__half_as_ushort( __float2half_rn( b ) ) << 16 );
}

__device__ __forceinline__ void st_f16x8( __half* __restrict__ p, size_t g, const float* v )
{
    *reinterpret_cast<uint4*>( p + g ) = make_uint4( pack2( v[0], v[1] ), pack2( v[2], v[3] ), pack2( v[4], v[5] ), pack2( v[6], v[7] ) );
}

// The fields a pass reads at its neighbours, for 8 cells of a row (Row) or one cell (One) of
// tile slot t, cell c: load() issues the loads (none for t < 0), value() forms the values, so
// that a lane's loads are all in flight before the first is waited for. t < 0 gives zeros.
struct FieldZ1  // down 1: the first sweep's z1 = w_A r' / d of the updated residual r - alpha q
{
    const uint16_t* code;
    const float* r0;
    const float* q;
    bool upd;  // r -= alpha q
    float alpha;
    float sc;
    const float* w;
    struct Row { uint4 c; float r[8], q[8]; };
    struct One { uint16_t c; float r, q; };
    __device__ __forceinline__ void load( Row& x, int t, int c ) const
    {
        x.c = make_uint4( 0u, 0u, 0u, 0u );
#pragma unroll
        for( int i = 0; i < 8; ++i ) x.r[i] = x.q[i] = 0.f;
        if( t < 0 ) return;
        const size_t g = (size_t)t * 512 + c;
        x.c = *reinterpret_cast<const uint4*>( code + g );
        bora_ld8( r0 + g, x.r );
        if( upd ) bora_ld8( q + g, x.q );
    }
    __device__ __forceinline__ void value( const Row& x, float* v ) const
    {
        uint16_t cc[8];
        codes8( x.c, cc );
#pragma unroll
        for( int i = 0; i < 8; ++i )
        {
            const float r = upd ? fmaf( -alpha, x.q[i], x.r[i] ) : x.r[i];
            v[i] = cfluid( cc[i] ) ? ( r * sc ) * w[cdiag( cc[i] )] : 0.f;
        }
    }
    __device__ __forceinline__ void load( One& x, int t, int c ) const
    {
        x.c = 0;
        x.r = x.q = 0.f;
        if( t < 0 ) return;
        const size_t g = (size_t)t * 512 + c;
        x.c = code[g];
        x.r = r0[g];
        if( upd ) x.q = q[g];
    }
    __device__ __forceinline__ float value( const One& x ) const
    {
        const float r = upd ? fmaf( -alpha, x.q, x.r ) : x.r;
        return cfluid( x.c ) ? ( r * sc ) * w[cdiag( x.c )] : 0.f;
    }
};

struct FieldF16  // down 2 and up 2: a scratch value stored in FP16
{
    const __half* v;
    struct Row { uint4 v; };
    struct One { __half v; };
    __device__ __forceinline__ void load( Row& x, int t, int c ) const
    {
        x.v = make_uint4( 0u, 0u, 0u, 0u );
        if( t >= 0 ) x.v = *reinterpret_cast<const uint4*>( v + (size_t)t * 512 + c );
    }
    __device__ __forceinline__ void value( const Row& x, float* o ) const { f16x8( x.v, o ); }
    __device__ __forceinline__ void load( One& x, int t, int c ) const
    {
        x.v = __half( 0.f );
        if( t >= 0 ) x.v = v[(size_t)t * 512 + c];
    }
    __device__ __forceinline__ float value( const One& x ) const { return __half2float( x.v ); }
};

struct FieldZa  // up 1: za = z0 + e(parent) on fluid cells
{
    const uint16_t* code;
    const __half* z0;
    const __half* ec;  // level 1's correction, 64 cells per tile
    struct Row { uint4 c, z; uint2 e; };
    struct One { uint16_t c; __half z, e; };
    __device__ __forceinline__ void load( Row& x, int t, int c ) const
    {
        x.c = x.z = make_uint4( 0u, 0u, 0u, 0u );
        x.e = make_uint2( 0u, 0u );
        if( t < 0 ) return;
        const size_t g = (size_t)t * 512 + c;
        const int jj = ( c >> 3 ) & 7, kk = c >> 6;
        x.c = *reinterpret_cast<const uint4*>( code + g );
        x.z = *reinterpret_cast<const uint4*>( z0 + g );
        x.e = *reinterpret_cast<const uint2*>( ec + (size_t)t * 64 + 4 * ( ( jj >> 1 ) + 4 * ( kk >> 1 ) ) );
    }
    __device__ __forceinline__ void value( const Row& x, float* v ) const
    {
        uint16_t cc[8];
        float zz[8];
        codes8( x.c, cc );
        f16x8( x.z, zz );
#pragma unroll
        for( int i = 0; i < 8; ++i )
        {
            const float ev = hbits( ( i >> 2 ) ? x.e.y : x.e.x, ( i >> 1 ) & 1 );
            v[i] = cfluid( cc[i] ) ? zz[i] + ev : 0.f;
        }
    }
    __device__ __forceinline__ void load( One& o, int t, int c ) const
    {
        o.c = 0;
        o.z = o.e = __half( 0.f );
        if( t < 0 ) return;
        const size_t g = (size_t)t * 512 + c;
        const int x = c & 7, jj = ( c >> 3 ) & 7, kk = c >> 6;
        o.c = code[g];
        o.z = z0[g];
        o.e = ec[(size_t)t * 64 + ( x >> 1 ) + 4 * ( ( jj >> 1 ) + 4 * ( kk >> 1 ) )];
    }
    __device__ __forceinline__ float value( const One& o ) const
    {
        return cfluid( o.c ) ? __half2float( o.z ) + __half2float( o.e ) : 0.f;
    }
};

// A half tile: the slots of its face neighbours (-1: none) and of the neighbour across its
// outer z face, its own slot, and which half (0: z layers 0..3, 1: 4..7).
struct HalfTile
{
    int smx, spx, smy, spy, sz, s, hi;
};

// The rows and cells around a lane's row that the warp's other lanes do not hold: the x ends,
// the y face row of lanes j = 0 / 7, and the z row below kk = 0 / above kk = 3 (the other half
// of the tile or the neighbour tile). load() before the values are needed, sums() from the
// lane's own values v (every lane of the warp calls both for the same half tile).
template <class F>
struct Around
{
    typename F::One xm, xp;
    typename F::Row y, z;
    __device__ __forceinline__ void load( const F& f, const HalfTile& h, int lane )
    {
        const int j = lane & 7, kk = lane >> 3, c = h.hi * 256 + 8 * lane;
        f.load( y, j == 0 ? h.smy : ( j == 7 ? h.spy : -1 ), c + ( j == 0 ? 56 : -56 ) );
        f.load( z, kk == 0 ? ( h.hi ? h.s : h.sz ) : ( kk == 3 ? ( h.hi ? h.sz : h.s ) : -1 ),
                8 * j + ( kk == 0 ? ( h.hi ? 192 : 448 ) : ( h.hi ? 0 : 256 ) ) );
        f.load( xm, h.smx, c + 7 );
        f.load( xp, h.spx, c );
    }
    __device__ __forceinline__ void sums( const F& f, int lane, const float* v, float* sum ) const
    {
        const int j = lane & 7, kk = lane >> 3;
        const float xl = f.value( xm ), xr = f.value( xp );
        float yh[8], zh[8];
        f.value( y, yh );
        f.value( z, zh );
#pragma unroll
        for( int i = 0; i < 8; ++i )
        {
            float ym = __shfl_up_sync( kAll, v[i], 1 ), yp = __shfl_down_sync( kAll, v[i], 1 );
            float zm = __shfl_up_sync( kAll, v[i], 8 ), zp = __shfl_down_sync( kAll, v[i], 8 );
            if( j == 0 ) ym = yh[i];
            if( j == 7 ) yp = yh[i];
            if( kk == 0 ) zm = zh[i];
            if( kk == 3 ) zp = zh[i];
            const float xm_ = i > 0 ? v[i > 0 ? i - 1 : 0] : xl, xp_ = i < 7 ? v[i < 7 ? i + 1 : 7] : xr;
            sum[i] = ( ( xm_ + xp_ ) + ( ym + yp ) ) + ( zm + zp );
        }
    }
};

struct Pass0Args
{
    BoraSolveTilesDev ft;
    BoraLevelDev F;       // level 0
    BoraLevelDev C;       // level 1 (down 2 writes its r; up 1 reads its z1)
    float* r0;            // the PCG residual (down 2 stores its update)
    const float* q;       // the PCG's A d (the update's direction term)
    float* scratch;       // FP32 per cell
    float* zout;          // up 2: the PCG's z
    BoraReduceDev red;
    int slot_rr;          // the scale's r.r
    int slot_rz_in, slot_dq_in;  // down 1, 2: alpha = rz_in / dq_in (slot_rz_in < 0: no update)
    int ndq;              // down 1: partial sums of dq to finish into slot_dq_in
};

// pass P of level 0: 0 = down 1, 1 = down 2, 2 = up 1, 3 = up 2; W half tiles (warps) per block
template <int W, int P>
__device__ __forceinline__ void pass0_body( const Pass0Args& a, unsigned bid, unsigned G )
{
    __shared__ float w[32];
    __shared__ float s_sc;
    bora_pdl_trigger();
    init_weights( w );
    const int lane = threadIdx.x & 31, j = lane & 7, kk = lane >> 3;
    const int nh = 2 * a.ft.n, stride = (int)G * W;
    // what no kernel of the solve writes - a half tile's table entry and its rows' codes - is
    // read one ahead, the first one's before the dependency wait
    HalfTile hn{ -1, -1, -1, -1, -1, 0, 0 };
    uint4 cwn = make_uint4( 0u, 0u, 0u, 0u );
    auto entry = [&]( int h ) {
        hn = HalfTile{ -1, -1, -1, -1, -1, 0, h & 1 };
        if( h >= nh ) return;
        const int4 n0 = __ldg( a.ft.tab + 2 * (size_t)( h >> 1 ) ), n1 = __ldg( a.ft.tab + 2 * (size_t)( h >> 1 ) + 1 );
        hn.smx = n0.x; hn.spx = n0.y; hn.smy = n0.z; hn.spy = n0.w;
        hn.sz = h & 1 ? n1.y : n1.x;
        hn.s = n1.z;
    };
    auto codes = [&]( int h ) {
        if( h < nh ) cwn = *reinterpret_cast<const uint4*>( a.F.code + (size_t)hn.s * 512 + hn.hi * 256 + 8 * lane );
    };
    int h = (int)bid * W + ( threadIdx.x >> 5 );
    entry( h );
    codes( h );
    __shared__ float2 s_dq[W];
    bora_pdl_wait();  // the previous kernel's results are complete from here
    if( threadIdx.x == 0 ) s_sc = residual_scale( a.red.ring[a.slot_rr] );
    const bool upd = ( P == 0 || P == 1 ) && a.slot_rz_in >= 0;  // down 1, 2 apply r -= alpha q
    float alpha = 0.f;
    if( P == 0 && upd )
    {
        const DF dq = part_collect( a.red.part_dq, a.ndq, s_dq );
        alpha = df_ratio( a.red.ringf[a.slot_rz_in], make_float2( dq.hi, dq.lo ) );
        if( bid == 0 && threadIdx.x == 0 ) ring_store( a.red, a.slot_dq_in, dq, false );
    }
    if( P == 1 && upd ) alpha = df_ratio( a.red.ringf[a.slot_rz_in], a.red.ringf[a.slot_dq_in] );
    __syncthreads();
    const float sc = s_sc, unscale = 1.f / sc;
    DF acc{ 0.f, 0.f };  // down 1: r.r of the updated residual; up 2: r.z
    __half* const scr = reinterpret_cast<__half*>( a.scratch );
    // the loop's bound is the block's, not the warp's: control flow that the compiler knows to be
    // uniform, without a reconvergence around each shuffle; a warp past the last half tile has no
    // neighbours and neither loads nor stores
#pragma unroll 1
    for( int base = (int)bid * W; base < nh; base += stride, h += stride )
    {
        const bool mine = h < nh;
        const HalfTile ht = hn;
        const int st = mine ? ht.s : -1, c0 = ht.hi * 256 + 8 * lane;
        const size_t g = (size_t)ht.s * 512 + c0;
        const uint4 cw = cwn;
        entry( h + stride );
        float r[8] = {}, q[8] = {}, v[8], sum[8];
        if( mine )
        {
            bora_ld8( a.r0 + g, r );
            if( upd ) bora_ld8( a.q + g, q );
        }
        uint16_t c[8];
        codes8( cw, c );
        auto update = [&]() {
            if( !upd ) return;
#pragma unroll
            for( int i = 0; i < 8; ++i ) r[i] = fmaf( -alpha, q[i], r[i] );
        };
        if constexpr( P == 0 )
        {
            const FieldZ1 f{ a.F.code, a.r0, a.q, upd, alpha, sc, w };
            Around<FieldZ1> ar;
            ar.load( f, ht, lane );
            update();
            float p = 0.f;
#pragma unroll
            for( int i = 0; i < 8; ++i ) p = fmaf( r[i], r[i], p );
            if( mine ) acc = df_add_f( acc, p );
#pragma unroll
            for( int i = 0; i < 8; ++i ) v[i] = cfluid( c[i] ) ? ( r[i] * sc ) * w[cdiag( c[i] )] : 0.f;
            ar.sums( f, lane, v, sum );
        }
        else if constexpr( P == 2 )
        {
            const FieldZa f{ a.F.code, a.F.z0, a.C.z1 };
            typename FieldZa::Row own;
            f.load( own, st, c0 );
            Around<FieldZa> ar;
            ar.load( f, ht, lane );
            f.value( own, v );
            ar.sums( f, lane, v, sum );
        }
        else
        {
            const FieldF16 f{ scr };
            typename FieldF16::Row own;
            f.load( own, st, c0 );
            Around<FieldF16> ar;
            ar.load( f, ht, lane );
            update();
            if( P == 1 && upd && mine ) bora_st8( a.r0 + g, r );
            if( P == 1 && mine ) *reinterpret_cast<uint4*>( a.F.z0 + g ) = own.v;  // z0 keeps z2
            f.value( own, v );
            ar.sums( f, lane, v, sum );
        }
        codes( h + stride );
        if constexpr( P == 0 || P == 2 )
        {
#pragma unroll
            for( int i = 0; i < 8; ++i ) v[i] = sweep( v[i], r[i] * sc, c[i], sum[i], w + 16 );
            if( mine ) st_f16x8( scr, g, v );
        }
        else if constexpr( P == 1 )
        {
            // the residual, restricted: x pairs in the row, y pairs from lane j + 1, z pairs from lane + 8
            float p[4];
#pragma unroll
            for( int i = 0; i < 8; ++i ) sum[i] = cfluid( c[i] ) ? r[i] * sc - ( (float)cdiag( c[i] ) * v[i] - sum[i] ) : 0.f;
#pragma unroll
            for( int i = 0; i < 4; ++i )
            {
                p[i] = sum[2 * i] + sum[2 * i + 1];
                p[i] = p[i] + __shfl_down_sync( kAll, p[i], 1 );
                p[i] = p[i] + __shfl_down_sync( kAll, p[i], 8 );
            }
            if( mine && !( j & 1 ) && !( kk & 1 ) )
                *reinterpret_cast<uint2*>( a.C.r + (size_t)ht.s * 64 + 4 * ( j >> 1 ) + 16 * ( 2 * ht.hi + ( kk >> 1 ) ) ) =
                    make_uint2( pack2( 0.5f * p[0], 0.5f * p[1] ), pack2( 0.5f * p[2], 0.5f * p[3] ) );
        }
        else
        {
            float trz = 0.f;
#pragma unroll
            for( int i = 0; i < 8; ++i )
            {
                v[i] = sweep( v[i], r[i] * sc, c[i], sum[i], w ) * unscale;  // undo the FP16 scaling of the residual
                if( cfluid( c[i] ) ) trz = fmaf( r[i], v[i], trz );
            }
            if( mine )
            {
                bora_st8( a.zout + g, v );
                acc = df_add_f( acc, trz );
            }
        }
    }
    if constexpr( P == 3 ) part_publish( acc, DF{ 0.f, 0.f }, a.red.part_rz, nullptr, bid );
    if constexpr( P == 0 ) part_publish( acc, DF{ 0.f, 0.f }, a.red.part_rr, nullptr, bid );
}

template <int W, int P>
__global__ void __launch_bounds__( 32 * W, pass_warps_per_sm( P ) / W ) k_mg_pass0( const __grid_constant__ Pass0Args a )
{
    pass0_body<W, P>( a, blockIdx.x, gridDim.x );
}

template <int W, int P>
__global__ void __launch_bounds__( 32 * W, pass_warps_per_sm( P ) / W ) k_mg_pass0_batch( const __grid_constant__ BoraBatchLaunch L )
{
    unsigned bid;
    const int k = bora_batch_member( L, blockIdx.x, &bid );
    const BoraMemberSolve& m = L.ms[k];
    const BoraMemberSlots& q = L.sl[k];
    Pass0Args a;
    a.ft = m.ft;
    a.F = m.L[0];
    a.C = m.L[1];
    a.r0 = m.sv.r;
    a.q = m.sv.q;
    a.scratch = m.sv.minv;
    a.zout = m.sv.z;
    a.red = m.red;
    a.slot_rr = q.rr;
    a.slot_rz_in = q.rz_in;
    a.slot_dq_in = q.dq_in;
    a.ndq = m.grid[kGridDir];
    pass0_body<W, P>( a, bid, (unsigned)m.grid[P == 0 || P == 3 ? kGridPass0R : kGridPass0] );
}

// ---- levels 1 and 2: one thread per x-row --------------------------------------------------

struct PassFArgs
{
    BoraSolveTilesDev ft;
    BoraLevelDev F;     // this level (E = 4 or 2)
    BoraLevelDev C;     // the coarser one (down 2 writes its r)
    const __half* ec;   // up 1: the coarser level's correction
    float* scratch;
};

// E 16-bit values in E / 2 words
template <int E>
__device__ __forceinline__ void ld16( const void* p, size_t g, uint32_t* w )
{
    const uint16_t* q = static_cast<const uint16_t*>( p ) + g;
    if constexpr( E == 4 )
    {
        const uint2 v = *reinterpret_cast<const uint2*>( q );
        w[0] = v.x;
        w[1] = v.y;
    }
    else w[0] = *reinterpret_cast<const uint32_t*>( q );
}
template <int E>
__device__ __forceinline__ void st16( __half* p, size_t g, const float* v )
{
    if constexpr( E == 4 ) *reinterpret_cast<uint2*>( p + g ) = make_uint2( pack2( v[0], v[1] ), pack2( v[2], v[3] ) );
    else *reinterpret_cast<uint32_t*>( p + g ) = pack2( v[0], v[1] );
}
__device__ __forceinline__ uint16_t word16( const uint32_t* w, int i ) { return (uint16_t)( w[i >> 1] >> ( 16 * ( i & 1 ) ) ); }

// pass P (0 = down 1, 1 = down 2, 2 = up 1, 3 = up 2) of a level with E = 4 or 2: a lane owns an
// x-row (j, k) of a tile, E * E lanes in a row of the warp own the tile. The neighbours in x are the
// lane's own, those in y and z other lanes' by shuffles, and the rows and cells across the tile's
// faces are loaded by the lanes at them. What no kernel of the solve writes - the table entry and
// the codes - is read before the dependency wait, so that it overlaps the previous kernel. (With
// a cell per thread, 235 instructions a cell at level 1: a V-cycle of 103 us at 256^3, 95 now, and
// of 244 us in a 640 tank of 16.8 K tiles, 220 now.)
template <int E, int P>
__device__ __forceinline__ void passf_body( const PassFArgs& a, unsigned bid )
{
    constexpr int R = E * E, E3 = E * E * E, H = E / 2, H3 = H * H * H, W = E / 2;
    constexpr bool kCodes = P == 0 || P == 2;  // the neighbours' values need their codes
    __shared__ float w[32];
    bora_pdl_trigger();
    init_weights( w );
    const size_t row = (size_t)bid * blockDim.x + threadIdx.x;
    const bool live = row < (size_t)a.ft.n * R;
    const int j = (int)( row % E ), k = (int)( row / E % E );
    const BoraLevelDev& F = a.F;
    int4 n0 = make_int4( -1, -1, -1, -1 ), n1 = n0;
    if( live )
    {
        n0 = __ldg( a.ft.tab + 2 * ( row / R ) );
        n1 = __ldg( a.ft.tab + 2 * ( row / R ) + 1 );
    }
    // a row of this level: its tile's slot (-1: none) and its j, k
    struct Row
    {
        int t, j, k;
        __device__ size_t at() const { return (size_t)t * E3 + E * ( j + E * k ); }
        __device__ size_t parent() const { return (size_t)t * H3 + H * ( ( j >> 1 ) + H * ( k >> 1 ) ); }
    };
    const Row own{ live ? n1.z : -1, j, k };
    const Row ry{ j == 0 ? n0.z : ( j == E - 1 ? n0.w : -1 ), j == 0 ? E - 1 : 0, k };
    const Row rz{ k == 0 ? n1.x : ( k == E - 1 ? n1.y : -1 ), j, k == 0 ? E - 1 : 0 };
    const Row rm{ live ? n0.x : -1, j, k }, rp{ live ? n0.y : -1, j, k };  // the x ends: the last / first cell
    uint32_t co[W] = {}, cy[W] = {}, cz[W] = {};
    uint16_t cm = 0, cp = 0;
    if( own.t >= 0 ) ld16<E>( F.code, own.at(), co );
    if constexpr( kCodes )
    {
        if( ry.t >= 0 ) ld16<E>( F.code, ry.at(), cy );
        if( rz.t >= 0 ) ld16<E>( F.code, rz.at(), cz );
        if( rm.t >= 0 ) cm = F.code[rm.at() + E - 1];
        if( rp.t >= 0 ) cp = F.code[rp.at()];
    }
    bora_pdl_wait();  // the previous kernel's results are complete from here
    __syncthreads();
    // the field that the pass reads at its neighbours: raw loads, then values
    struct Raw
    {
        uint32_t h[W], e;  // residual or z0; the parents' correction
        float f[E];        // scratch
    };
    auto load = [&]( const Row& r, Raw& x ) {
#pragma unroll
        for( int i = 0; i < W; ++i ) x.h[i] = 0u;
        x.e = 0u;
#pragma unroll
        for( int i = 0; i < E; ++i ) x.f[i] = 0.f;
        if( r.t < 0 ) return;
        if constexpr( P == 0 ) ld16<E>( F.r, r.at(), x.h );
        else if constexpr( P == 2 )
        {
            ld16<E>( F.z0, r.at(), x.h );
            if constexpr( H == 2 ) x.e = *reinterpret_cast<const uint32_t*>( a.ec + r.parent() );
            else x.e = *reinterpret_cast<const uint16_t*>( a.ec + r.parent() );
        }
        else if constexpr( E == 4 )
        {
            const float4 v = *reinterpret_cast<const float4*>( a.scratch + r.at() );
            x.f[0] = v.x; x.f[1] = v.y; x.f[2] = v.z; x.f[3] = v.w;
        }
        else
        {
            const float2 v = *reinterpret_cast<const float2*>( a.scratch + r.at() );
            x.f[0] = v.x; x.f[1] = v.y;
        }
    };
    auto value = [&]( const Raw& x, uint16_t c, int i ) -> float {
        if constexpr( P == 0 ) return cfluid( c ) ? hbits( x.h[i >> 1], i & 1 ) * w[cdiag( c )] : 0.f;
        else if constexpr( P == 2 ) return cfluid( c ) ? hbits( x.h[i >> 1], i & 1 ) + hbits( x.e, i >> 1 ) : 0.f;
        else return x.f[i];
    };
    auto one = [&]( const Row& r, uint16_t c, int i ) -> float {
        if( r.t < 0 ) return 0.f;
        if constexpr( P == 0 ) return cfluid( c ) ? __half2float( F.r[r.at() + i] ) * w[cdiag( c )] : 0.f;
        else if constexpr( P == 2 ) return cfluid( c ) ? __half2float( F.z0[r.at() + i] ) + __half2float( a.ec[r.parent() + ( i >> 1 )] ) : 0.f;
        else return a.scratch[r.at() + i];
    };
    Raw xo, xy, xz;
    load( own, xo );
    load( ry, xy );
    load( rz, xz );
    const float xm = one( rm, cm, E - 1 ), xp = one( rp, cp, 0 );
    uint32_t rw[W] = {};
    if( own.t >= 0 ) ld16<E>( F.r, own.at(), rw );
    float v[E], out[E];
#pragma unroll
    for( int i = 0; i < E; ++i ) v[i] = value( xo, word16( co, i ), i );
#pragma unroll
    for( int i = 0; i < E; ++i )
    {
        const uint16_t c = word16( co, i );
        float ym = __shfl_up_sync( kAll, v[i], 1 ), yp = __shfl_down_sync( kAll, v[i], 1 );
        float zm = __shfl_up_sync( kAll, v[i], E ), zp = __shfl_down_sync( kAll, v[i], E );
        const float hy = value( xy, word16( cy, i ), i ), hz = value( xz, word16( cz, i ), i );
        if( j == 0 ) ym = hy;
        if( j == E - 1 ) yp = hy;
        if( k == 0 ) zm = hz;
        if( k == E - 1 ) zp = hz;
        const float sum = ( ( ( i ? v[i ? i - 1 : 0] : xm ) + ( i < E - 1 ? v[i < E - 1 ? i + 1 : 0] : xp ) ) + ( ym + yp ) ) + ( zm + zp );
        const float r = cfluid( c ) ? hbits( rw[i >> 1], i & 1 ) : 0.f;
        if constexpr( P == 1 ) out[i] = cfluid( c ) ? r - ( (float)cdiag( c ) * v[i] - sum ) : 0.f;
        else out[i] = sweep( v[i], r, c, sum, P == 3 ? w : w + 16 );
    }
    if constexpr( P == 1 )
    {
        // restriction: x pairs in the row, y pairs from lane j + 1, z pairs from lane + E
        float q[2];
#pragma unroll
        for( int i = 0; i < H; ++i )
        {
            q[i] = out[2 * i] + out[2 * i + 1];
            q[i] = q[i] + __shfl_down_sync( kAll, q[i], 1 );
            q[i] = q[i] + __shfl_down_sync( kAll, q[i], E );
        }
        if( own.t >= 0 && !( j & 1 ) && !( k & 1 ) )
        {
            if constexpr( H == 2 ) *reinterpret_cast<uint32_t*>( a.C.r + own.parent() ) = pack2( 0.5f * q[0], 0.5f * q[1] );
            else a.C.r[own.parent()] = __float2half_rn( 0.5f * q[0] );
        }
    }
    if( own.t < 0 ) return;
    if constexpr( P == 1 ) st16<E>( F.z0, own.at(), v );
    else if constexpr( P == 3 ) st16<E>( F.z1, own.at(), out );
    else if constexpr( E == 4 ) *reinterpret_cast<float4*>( a.scratch + own.at() ) = make_float4( out[0], out[1], out[2], out[3] );
    else *reinterpret_cast<float2*>( a.scratch + own.at() ) = make_float2( out[0], out[1] );
}

template <int E, int P, int T>
__global__ void __launch_bounds__( T ) k_mg_passf( const __grid_constant__ PassFArgs a )
{
    passf_body<E, P>( a, blockIdx.x );
}

template <int E, int P, int T>
__global__ void __launch_bounds__( T ) k_mg_passf_batch( const __grid_constant__ BoraBatchLaunch L )
{
    constexpr int l = E == 4 ? 1 : 2;
    unsigned bid;
    const int k = bora_batch_member( L, blockIdx.x, &bid );
    const BoraMemberSolve& m = L.ms[k];
    PassFArgs a;
    a.ft = m.ft;
    a.F = m.L[l];
    a.C = m.L[l + 1];
    a.ec = l == 1 ? m.L[2].z1 : m.z3;
    a.scratch = m.sv.minv;
    passf_body<E, P>( a, bid );
}

int num_sms_pass()
{
    static BoraPerDevice sms;
    return sms.get( [] {
        int dev = 0, n = 0;
        cudaGetDevice( &dev );
        cudaDeviceGetAttribute( &n, cudaDevAttrMultiProcessorCount, dev );
        return n > 0 ? n : 152;
    } );
}

template <int E, int P>
void launch_passf( const PassFArgs& a, int v, cudaStream_t st )
{
    const int g = bora_mg_pass_grid( E, a.ft.n, v );
    if( g <= 0 ) return;
    switch( v )
    {
    case 0: bora_launch_pdl( k_mg_passf<E, P, 64>, dim3( g ), dim3( 64 ), 0, st, a ); break;
    case 1: bora_launch_pdl( k_mg_passf<E, P, 128>, dim3( g ), dim3( 128 ), 0, st, a ); break;
    case 2: bora_launch_pdl( k_mg_passf<E, P, 256>, dim3( g ), dim3( 256 ), 0, st, a ); break;
    default: bora_launch_pdl( k_mg_passf<E, P, 512>, dim3( g ), dim3( 512 ), 0, st, a ); break;
    }
}

template <int P>
void launch_pass0( const Pass0Args& a, int v, cudaStream_t st )
{
    const int g = bora_mg_pass_grid( 8, a.ft.n, v );
    if( g <= 0 ) return;
    switch( v )
    {
    case 0: bora_launch_pdl( k_mg_pass0<2, P>, dim3( g ), dim3( 64 ), 0, st, a ); break;
    case 1: bora_launch_pdl( k_mg_pass0<4, P>, dim3( g ), dim3( 128 ), 0, st, a ); break;
    default: bora_launch_pdl( k_mg_pass0<8, P>, dim3( g ), dim3( 256 ), 0, st, a ); break;
    }
}

}  // namespace

// Grid of the passes of a level with E cells per tile edge in launch shape v: level 0 as many
// blocks as make equal rounds of warps over the half tiles with the warps per SM that its
// registers allow (v < 0: the reducing passes, at most kBoraMaxReduceBlocks); levels 1 and 2
// one thread per x-row.
int bora_mg_pass_grid( int E, int ntiles, int v )
{
    if( ntiles <= 0 ) return 0;
    const int sms = num_sms_pass();
    if( E == 8 )
    {
        const int W = v < 0 ? kReduceWarps : kPassWarpsOf[std::min( v, 2 )];
        const int cap = std::max( 1, std::min( ( v < 0 ? kReduceWarpsPerSm : kPassWarpsPerSm ) / W * sms, kBoraMaxReduceBlocks ) ) * W;
        const int rounds = ( 2 * ntiles + cap - 1 ) / cap;
        return std::max( 1, ( 2 * ntiles + W * rounds - 1 ) / ( W * rounds ) );
    }
    const int T = kFlatThreadsOf[std::min( std::max( v, 0 ), 3 )];
    const size_t n = (size_t)ntiles * E * E;
    return (int)( ( n + T - 1 ) / T );
}

void bora_mg_pass_down( const BoraLevelDev* levels, int l, const BoraSolveTilesDev& t, float* r0, const float* q,
                        float* scratch, const BoraReduceDev& red, int slot_rr, int slot_rz_in, int slot_dq_in,
                        cudaStream_t st )
{
    const int group = l == 0 ? kBoraTuneL0 : ( l == 1 ? kBoraTuneL1 : kBoraTuneL2 );
    const BoraTunePick pick = bora_tune_pick( group, t.n );
    BoraTuneTimer timer( pick, group, t.n, st );  // times the level's two down passes
    const int v = pick.variant;
    if( levels[l].E == 8 )
    {
        Pass0Args a{};
        a.ft = t; a.F = levels[0]; a.C = levels[1]; a.r0 = r0; a.q = q; a.scratch = scratch;
        a.red = red; a.slot_rr = slot_rr;
        a.slot_rz_in = slot_rz_in; a.slot_dq_in = slot_dq_in; a.ndq = bora_pcg_direction_grid( t.n );
        // down 1 sums r.r over its blocks: the fixed shape
        const int g = bora_mg_pass_grid( 8, t.n, -1 );
        if( g > 0 ) bora_launch_pdl( k_mg_pass0<kReduceWarps, 0>, dim3( g ), dim3( 32 * kReduceWarps ), 0, st, a );
        launch_pass0<1>( a, v, st );
        return;
    }
    PassFArgs a{};
    a.ft = t; a.F = levels[l]; a.C = levels[l + 1]; a.scratch = scratch;
    if( levels[l].E == 4 ) { launch_passf<4, 0>( a, v, st ); launch_passf<4, 1>( a, v, st ); }
    else { launch_passf<2, 0>( a, v, st ); launch_passf<2, 1>( a, v, st ); }
}

void bora_mg_pass_up( const BoraLevelDev* levels, int l, const __half* ec, const BoraSolveTilesDev& t, const float* r0,
                      float* scratch, const BoraReduceDev& red, int slot_rr, float* z, cudaStream_t st )
{
    const int group = l == 0 ? kBoraTuneL0 : ( l == 1 ? kBoraTuneL1 : kBoraTuneL2 );
    const int v = bora_tune_pick( group, t.n ).variant;
    if( levels[l].E == 8 )
    {
        Pass0Args a{};
        a.ft = t; a.F = levels[0]; a.C = levels[1]; a.C.z1 = const_cast<__half*>( ec );
        a.r0 = const_cast<float*>( r0 ); a.scratch = scratch; a.zout = z; a.red = red; a.slot_rr = slot_rr;
        a.slot_rz_in = -1; a.slot_dq_in = -1;
        launch_pass0<2>( a, v, st );
        // r.z: the fixed shape
        const int g = bora_mg_pass_grid( 8, t.n, -1 );
        if( g > 0 ) bora_launch_pdl( k_mg_pass0<kReduceWarps, 3>, dim3( g ), dim3( 32 * kReduceWarps ), 0, st, a );
        return;
    }
    PassFArgs a{};
    a.ft = t; a.F = levels[l]; a.C = levels[l + 1]; a.ec = ec; a.scratch = scratch;
    if( levels[l].E == 4 ) { launch_passf<4, 2>( a, v, st ); launch_passf<4, 3>( a, v, st ); }
    else { launch_passf<2, 2>( a, v, st ); launch_passf<2, 3>( a, v, st ); }
}

void bora_launch_mg_pass_batch( int l, int pass, int v, const BoraBatchLaunch& L, int blocks, cudaStream_t st )
{
    if( blocks <= 0 ) return;
    const dim3 grid( blocks );
    if( l == 0 )
    {
        // down 1 and up 2 reduce over their blocks: the fixed shape
        if( pass == 0 || pass == 3 )
        {
            if( pass == 0 ) bora_launch_pdl( k_mg_pass0_batch<kReduceWarps, 0>, grid, dim3( 32 * kReduceWarps ), 0, st, L );
            else bora_launch_pdl( k_mg_pass0_batch<kReduceWarps, 3>, grid, dim3( 32 * kReduceWarps ), 0, st, L );
            return;
        }
        const int W = kPassWarpsOf[std::min( std::max( v, 0 ), 2 )];
        const dim3 blk( 32 * W );
        auto go = [&]( auto k1, auto k2 ) {
            if( pass == 1 ) bora_launch_pdl( k1, grid, blk, 0, st, L );
            else bora_launch_pdl( k2, grid, blk, 0, st, L );
        };
        if( W == 2 ) go( k_mg_pass0_batch<2, 1>, k_mg_pass0_batch<2, 2> );
        else if( W == 4 ) go( k_mg_pass0_batch<4, 1>, k_mg_pass0_batch<4, 2> );
        else go( k_mg_pass0_batch<8, 1>, k_mg_pass0_batch<8, 2> );
        return;
    }
    const int T = kFlatThreadsOf[std::min( std::max( v, 0 ), 3 )];
    auto flat = [&]( auto tag ) {
        constexpr int E = decltype( tag )::value;
        auto go = [&]( auto k0, auto k1, auto k2, auto k3 ) {
            const dim3 blk( T );
            if( pass == 0 ) bora_launch_pdl( k0, grid, blk, 0, st, L );
            else if( pass == 1 ) bora_launch_pdl( k1, grid, blk, 0, st, L );
            else if( pass == 2 ) bora_launch_pdl( k2, grid, blk, 0, st, L );
            else bora_launch_pdl( k3, grid, blk, 0, st, L );
        };
        if( T == 64 ) go( k_mg_passf_batch<E, 0, 64>, k_mg_passf_batch<E, 1, 64>, k_mg_passf_batch<E, 2, 64>, k_mg_passf_batch<E, 3, 64> );
        else if( T == 128 ) go( k_mg_passf_batch<E, 0, 128>, k_mg_passf_batch<E, 1, 128>, k_mg_passf_batch<E, 2, 128>, k_mg_passf_batch<E, 3, 128> );
        else if( T == 256 ) go( k_mg_passf_batch<E, 0, 256>, k_mg_passf_batch<E, 1, 256>, k_mg_passf_batch<E, 2, 256>, k_mg_passf_batch<E, 3, 256> );
        else go( k_mg_passf_batch<E, 0, 512>, k_mg_passf_batch<E, 1, 512>, k_mg_passf_batch<E, 2, 512>, k_mg_passf_batch<E, 3, 512> );
    };
    if( l == 1 ) flat( std::integral_constant<int, 4>{} );
    else flat( std::integral_constant<int, 2>{} );
}
