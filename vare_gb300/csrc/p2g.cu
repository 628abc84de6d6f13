// P2G on the sparse grid, fused with the particle-count field and the cell flags.
//
// Replaces Rasterization::PointsToVelField / PointsToCountField (sparse,
// base/source/Rasterization.cu:122-229), which scatter with 4 (+1) float atomics per
// stencil cell per particle, and the flags lambda of FLIPMethod::advanceOneStep
// (base/source/FLIPMethod.cu:242-281).
//
// Particles arrive sorted by dual cell (the base cell of the reference's 2x2x2 stencil,
// max(int(p-0.5),0) per axis), so the particles that touch cell c are exactly those of
// the 8 dual cells {c-1, c}^3. Each dual cell's particles are read once and summed per
// stencil corner, and each cell adds its 8 corner sums - no atomics, one store per field.
// Weights follow the reference (w = prod max(0, 1-|p-c|) + 1e-5); sums are FP32 in a
// fixed order (particles of a dual cell by source index, then a fixed tree over the 8
// dual cells), so the result is bit-reproducible.
#include "bora_internal.h"

namespace {

// Collider velocity at a cell centre (FLIPMethod.cu:248,260), out of line: rare, and its
// corner arrays would otherwise raise the register count of the whole kernel.
__device__ __noinline__ float3 col_velocity( const BoraGridDev* g, float x, float y, float z )
{
    float cv[3];
    bora_col_lerp( g->cols, g->nx, g->ny, g->nz, x, y, z, 2, cv );
    return make_float3( cv[0], cv[1], cv[2] );
}

// Whether a collider value at the centre of a cell of tile (ti, tj, tk) can be negative. The
// values are lerps of samples at cell centres within 4.5 cells of the tile's centre per axis. A
// box's distance changes by at most the distance moved, so a tile whose centre is 8 cells or more
// from every box has positive samples only; a sparse collider's samples are its (positive)
// background where neither the tile nor one next to it holds a collider tile.
__device__ inline bool col_near( const BoraGridDev& g, int ti, int tj, int tk )
{
    if( g.cols.tslot ) return !( g.cols.tbg > 0.f ) || g.cols.tnear[(size_t)ti + (size_t)g.tx * ( (size_t)tj + (size_t)g.ty * tk )];
    if( g.cols.fphi || !( g.cols.band > 0.f ) ) return true;
    const float x = (float)( ti * BORA_TILE + 4 ), y = (float)( tj * BORA_TILE + 4 ), z = (float)( tk * BORA_TILE + 4 );
    for( int n = 0; n < g.cols.count; ++n )
        if( !( bora_box_sdf( g.cols.box[n], x, y, z ) > 8.f ) ) return true;
    return false;
}

// One CTA per tile, over the 9^3 dual cells (tile-local coordinates -1 .. 7) that touch it: a
// lane takes one dual cell, a warp three x-rows of nine at a time. A lane reads its dual cell's
// particles once in bin order (fixed by k_order_bins) and keeps the 8 corner sums of m, m*v in
// registers; the two dual cells that share a face in x lie in adjacent lanes, so their corner
// sums are added by a shuffle, and the four sums a cell gets per value (two in y, two in z) are
// parked in shared memory by exactly one lane each and added by a fixed tree, so the result is
// reproducible. Halo dual cells are recomputed by every tile that needs them instead of being
// exchanged.
//
// The loop over a dual cell's particles is bound by L1: a load instruction touches the lines of
// three rows (8 or 9 of them), and what 27 warps have in flight (163 KB) does not fit it. So:
// the next particle is loaded ahead, x-adjacent corners are packed pairs (two FP32 operations an
// instruction), the shared memory is 36 KB (three CTAs of 9 warps, the
// rest of the 256 KB is L1), and the collider code, whose calls spilled the loop's registers,
// is another kernel. At 256^3 (24.6 M particles, 8.2 K tiles) 546 -> 432 us; a 640 tank with a
// collider 1120 -> 775 us (its samples only in tiles near it). Slower: two CTAs of 9 or of 14
// warps (483, 488), five of 5 (676), particles staged in shared memory four ranks at a time by
// asynchronous copies (457 with two CTAs; 792 with three, L1 then holds 47 KB), batches of two
// particles in registers (475).
constexpr int kP2GThreads = 288;  // 9 warps: the 27 groups of three rows in three rounds
constexpr int kP2GEdge = BORA_TILE + 1;
constexpr size_t kP2GSmem = 4 * 4 * 512 * sizeof( float ) + kP2GEdge * kP2GEdge * kP2GEdge * sizeof( uint32_t );

__device__ __forceinline__ float2 mul2( float2 a, float2 b ) { return __fmul2_rn( a, b ); }
__device__ __forceinline__ float2 add2( float2 a, float2 b ) { return __fadd2_rn( a, b ); }

// COL: there are colliders (their code is large and its calls cost the loop registers).
template <bool COL>
__global__ void __launch_bounds__( kP2GThreads, 3 ) k_p2g( const __grid_constant__ BoraGridDev g, BoraTilesDev t,
                                                           BoraParticlesDev p, const uint32_t* __restrict__ idx,
                                                           const uint32_t* __restrict__ start, BoraCellsDev c )
{
    extern __shared__ float p2g_smem[];
    float* part = p2g_smem;  // [y, z source][m, mx, my, mz][cell]
    uint32_t* pcnt = reinterpret_cast<uint32_t*>( p2g_smem + 4 * 4 * 512 );  // [dual cell]
    __shared__ int32_t nb[27];
    const int s = blockIdx.x, tid = threadIdx.x, lane = tid & 31;
    if( tid < 27 ) nb[tid] = t.nbr[(size_t)s * 27 + tid];
    const int vt = t.tile_of[s];
    const int ti = vt % g.tx, tj = ( vt / g.tx ) % g.ty, tk = vt / ( g.tx * g.ty );
    __syncthreads();
    const int di = lane % 9 - 1;  // tile-local dual-cell coordinates in [-1, 7]
#pragma unroll 1
    for( int item = tid >> 5; item < 27; item += kP2GThreads / 32 )
    {
        const int dj = 3 * ( item % 3 ) + lane / 9 - 1, dk = item / 3 - 1;
        const int ns = lane < 27 ? nb[bora_dir( di < 0 ? -1 : 0, dj < 0 ? -1 : 0, dk < 0 ? -1 : 0 )] : -1;
        uint32_t q0 = 0, q1 = 0;
        if( ns >= 0 )
        {
            const uint32_t key = (uint32_t)ns * BORA_TILE_CELLS + (uint32_t)bora_local( di, dj, dk );
            q0 = start[key];
            q1 = start[key + 1];
        }
        // centres of the two cells per axis that the dual cell's particles touch
        const int gi = ti * BORA_TILE + di, gj = tj * BORA_TILE + dj, gk = tk * BORA_TILE + dk;
        const float cx0 = (float)gi + .5f, cx1 = (float)( gi + 1 ) + .5f;
        const float cy0 = (float)gj + .5f, cy1 = (float)( gj + 1 ) + .5f;
        const float cz0 = (float)gk + .5f, cz1 = (float)( gk + 1 ) + .5f;
        // corners (0, b, c) and (1, b, c) as a pair, [b + 2 c][m, mx, my, mz]
        float2 acc[4][4];
#pragma unroll
        for( int o = 0; o < 4; ++o ) acc[o][0] = acc[o][1] = acc[o][2] = acc[o][3] = make_float2( 0.f, 0.f );
        // a particle is loaded while the one before is summed, its index two ahead
        float xn = 0.f, yn = 0.f, zn = 0.f, vxn = 0.f, vyn = 0.f, vzn = 0.f;
        uint32_t in = 0;
        auto fetch = [&]( uint32_t pi ) {
            xn = p.px[pi]; yn = p.py[pi]; zn = p.pz[pi];
            vxn = p.vx[pi]; vyn = p.vy[pi]; vzn = p.vz[pi];
        };
        if( q0 < q1 ) fetch( idx[q0] );
        if( q0 + 1 < q1 ) in = idx[q0 + 1];
#pragma unroll 1
        for( uint32_t q = q0; q < q1; ++q )
        {
            const float x = xn, y = yn, z = zn, vx = vxn, vy = vyn, vz = vzn;
            if( q + 1 < q1 )
            {
                fetch( in );
                if( q + 2 < q1 ) in = idx[q + 2];
            }
            const float2 wx = make_float2( fmaxf( 0.f, 1.f - fabsf( x - cx0 ) ), fmaxf( 0.f, 1.f - fabsf( x - cx1 ) ) );
            const float wy[2] = { fmaxf( 0.f, 1.f - fabsf( y - cy0 ) ), fmaxf( 0.f, 1.f - fabsf( y - cy1 ) ) };
            const float wz[2] = { fmaxf( 0.f, 1.f - fabsf( z - cz0 ) ), fmaxf( 0.f, 1.f - fabsf( z - cz1 ) ) };
            // weights and their products with the velocity with fused multiply-adds: one rounding
            // fewer than the reference's (whose atomics add in no fixed order)
            const float2 wxy[2] = { mul2( wx, make_float2( wy[0], wy[0] ) ), mul2( wx, make_float2( wy[1], wy[1] ) ) };
#pragma unroll
            for( int o = 0; o < 4; ++o )
            {
                const float2 w = __ffma2_rn( wxy[o & 1], make_float2( wz[o >> 1], wz[o >> 1] ), make_float2( 1e-05f, 1e-05f ) );
                acc[o][0] = add2( acc[o][0], w );
                acc[o][1] = __ffma2_rn( w, make_float2( vx, vx ), acc[o][1] );
                acc[o][2] = __ffma2_rn( w, make_float2( vy, vy ), acc[o][2] );
                acc[o][3] = __ffma2_rn( w, make_float2( vz, vz ), acc[o][3] );
            }
        }
        if( lane < 27 ) pcnt[item * 27 + lane] = q1 - q0;
        // cell (di, dj + b, dk + c): the corner x = 1 of dual cell di - 1 plus the own corner x = 0
#pragma unroll
        for( int o = 0; o < 4; ++o )
        {
            const int lj = dj + ( o & 1 ), lk = dk + ( o >> 1 );
            const bool in_tile = lane < 27 && di >= 0 && lj >= 0 && lk >= 0 && lj < 8 && lk < 8;
            const int at = ( 3 - o ) * 4 * 512 + ( di | ( lj << 3 ) | ( lk << 6 ) );
#pragma unroll
            for( int v = 0; v < 4; ++v )
            {
                const float below = __shfl_up_sync( 0xffffffffu, acc[o][v].y, 1 );
                if( in_tile ) part[at + v * 512] = below + acc[o][v].x;
            }
        }
    }
    __syncthreads();
    const bool near_col = COL && col_near( g, ti, tj, tk );
    // per cell: fixed tree over the sums of its 8 source dual cells (x pairs are added already)
    for( int l = tid; l < BORA_TILE_CELLS; l += kP2GThreads )
    {
        auto tree = [&]( int v ) {
            const float* q = part + v * 512 + l;
            return ( q[0 * 2048] + q[1 * 2048] ) + ( q[2 * 2048] + q[3 * 2048] );
        };
        const float m = tree( 0 ), mx = tree( 1 ), my = tree( 2 ), mz = tree( 3 );
        uint32_t cnt = 0;
        {
            const uint32_t* n = pcnt + ( l & 7 ) + kP2GEdge * ( ( ( l >> 3 ) & 7 ) + kP2GEdge * ( l >> 6 ) );
#pragma unroll
            for( int o = 0; o < 8; ++o ) cnt += n[( o & 1 ) + kP2GEdge * ( ( ( o >> 1 ) & 1 ) + kP2GEdge * ( o >> 2 ) )];
        }
        const size_t cell = (size_t)s * BORA_TILE_CELLS + l;
        const int i = ti * BORA_TILE + ( l & 7 ), j = tj * BORA_TILE + ( ( l >> 3 ) & 7 ), k = tk * BORA_TILE + ( l >> 6 );
        if( !( i < g.nx && j < g.ny && k < g.nz ) )
        {
            c.flag[cell] = BORA_MASKED;
            c.mass[cell] = 0.f; c.surf[cell] = 0.f;
            c.vx[cell] = 0.f; c.vy[cell] = 0.f; c.vz[cell] = 0.f;
            continue;
        }
        float vx = 0.f, vy = 0.f, vz = 0.f, mass = 0.f;
        if( m > 0.f )
        {
            mass = m;
            vx = mx / m;
            vy = my / m;
            vz = mz / m;
        }
        // flags and collider velocity (FLIPMethod.cu:244-260)
        uint8_t f = m > 0.f ? BORA_FLUID : BORA_AIR;
        if constexpr( COL )
        {
            const float ccx = (float)i + .5f, ccy = (float)j + .5f, ccz = (float)k + .5f;
            if( near_col && bora_col_phi( g, ccx, ccy, ccz ) < 0.f )
            {
                if( !( m > 0.f ) ) f = BORA_SOLID;
                const float3 cv = col_velocity( &g, ccx, ccy, ccz );
                vx += cv.x * g.col_vel_scale;
                vy += cv.y * g.col_vel_scale;
                vz += cv.z * g.col_vel_scale;
            }
        }
        c.flag[cell] = f;
        c.mass[cell] = mass;
        c.surf[cell] = (float)cnt;
        c.vx[cell] = vx;
        c.vy[cell] = vy;
        c.vz[cell] = vz;
    }
}

}  // namespace

void bora_launch_p2g( const BoraGridDev& g, int ntiles, BoraTilesDev t, BoraParticlesDev p, const uint32_t* idx,
                      const uint32_t* start, BoraCellsDev c, cudaStream_t st )
{
    if( ntiles <= 0 ) return;
    static BoraPerDevice attr_set;
    attr_set.get( [] {
        cudaFuncSetAttribute( k_p2g<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kP2GSmem );
        cudaFuncSetAttribute( k_p2g<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kP2GSmem );
        return 1;
    } );
    if( bora_col_active( g.cols ) ) k_p2g<true><<<ntiles, kP2GThreads, kP2GSmem, st>>>( g, t, p, idx, start, c );
    else k_p2g<false><<<ntiles, kP2GThreads, kP2GSmem, st>>>( g, t, p, idx, start, c );
}
