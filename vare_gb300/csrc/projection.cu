// Pressure projection over active 8^3 tiles: right-hand side and stencil build, a
// matrix-free PCG with a block-MIC(0) preconditioner, FP64-accurate (double-float)
// reductions and double-float iterative refinement, and the pressure-gradient velocity
// update.
//
// Replaces FluidProjection::buildLinearSystem / solve (sparse,
// base/source/FluidProjection.cu:165-381), LinearSystemSolver::cg/pcg
// (base/source/LinearSystemSolver.cpp:12-105) and the BLAS kernels they call
// (base/source/BLAS.cu:12-331). The reference assembles a 7-entry ELL matrix
// (float values + size_t columns, 84 B per row) after a serial host relabel of the
// fluid cells; here the operator is applied from a 16-bit per-cell stencil code
// (neighbour-is-fluid mask + integer diagonal), which encodes the same matrix.
#include <algorithm>

#include "bora_internal.h"
#include "half_rows.cuh"
#include "reduce.cuh"

namespace {

__device__ inline float absr( float x ) { return x < 0.f ? -x : x; }  // MathUtils.h:129 Abs

// ---------------------------------------------------------------------------------
// The row stencils (half_rows.cuh) of the right-hand side and the velocity update.
// Half tiles per CTA: 4 (the system's build 94.7 us, of which the right-hand side is 35, the velocity update
// 44.5 at 256^3; 102 and 53 with 8)
constexpr int kRowWarps = 4;

__device__ __forceinline__ uint2 flags8( const uint8_t* __restrict__ flag, int t, int c )
{
    return t < 0 ? make_uint2( 0u, 0u ) : *reinterpret_cast<const uint2*>( flag + (size_t)t * BORA_TILE_CELLS + c );  // BORA_AIR is 0
}
__device__ __forceinline__ int flag_of( uint2 w, int i ) { return (int)( ( ( i < 4 ? w.x : w.y ) >> ( 8 * ( i & 3 ) ) ) & 255u ); }

__device__ __forceinline__ uint2 shfl2( uint2 w, int lane )
{
    return make_uint2( __shfl_sync( 0xffffffffu, w.x, lane ), __shfl_sync( 0xffffffffu, w.y, lane ) );
}

// A row's flags and those of the rows around it in y and z, and at its x ends. A cell beyond the grid
// (the frame's extents are multiples of 4, so half a row or all of it) is air, whatever flag the
// caller may have set there.
struct RowFlags
{
    uint2 w, ym, yp, zm, zp;
    int xm, xp;
    bool in_grid[2];  // the row's cells 0..3, 4..7
    __device__ __forceinline__ void load( const BoraGridDev& g, const uint8_t* __restrict__ flag, const HalfRow& r )
    {
        const int lane = threadIdx.x & 31;
        w = flags8( flag, r.mine ? r.s : -1, r.c );
        in_grid[0] = r.J < g.ny && r.K < g.nz;
        in_grid[1] = in_grid[0] && r.i0 + 4 < g.nx;
        w = make_uint2( in_grid[0] ? w.x : 0u, in_grid[1] ? w.y : 0u );
        const uint2 y = flags8( flag, r.yt, r.yc ), z = flags8( flag, r.zt, r.zc );
        xm = r.xm < 0 ? BORA_AIR : flag[(size_t)r.xm * BORA_TILE_CELLS + r.c + 7];
        xp = r.xp < 0 ? BORA_AIR : flag[(size_t)r.xp * BORA_TILE_CELLS + r.c];
        ym = shfl2( w, lane - 1 ); yp = shfl2( w, lane + 1 );
        zm = shfl2( w, lane - 8 ); zp = shfl2( w, lane + 8 );
        if( r.j == 0 ) ym = y;
        if( r.j == 7 ) yp = y;
        if( r.kk == 0 ) zm = z;
        if( r.kk == 3 ) zp = z;
    }
};

// ---------------------------------------------------------------------------------
// Right-hand side and stencil code (FluidProjection.cu:203-266). (With a cell per thread from a
// staged 10^3 region it was bound by index arithmetic: 84 us at 256^3, 35 now.)
__global__ void __launch_bounds__( 32 * kRowWarps ) k_rhs( BoraGridDev g, BoraTilesDev t, int ntiles, BoraCellsDev c,
                                                           uint32_t* nfluid, uint8_t* __restrict__ tile_fluid )
{
    __shared__ int any[kRowWarps];
    const HalfRow r = half_row<kRowWarps>( g, t, ntiles );
    RowFlags f;
    f.load( g, c.flag, r );
    const int own = r.mine ? r.s : -1;
    float vx[8], vy[8], vz[8], vym[8], vyp[8], vzm[8], vzp[8], yh[8], zh[8];
    row8( c.vx, own, r.c, vx );
    row8( c.vy, own, r.c, vy );
    row8( c.vz, own, r.c, vz );
    row8( c.vy, r.yt, r.yc, yh );
    row8( c.vz, r.zt, r.zc, zh );
    const float vxm = r.xm < 0 ? 0.f : c.vx[(size_t)r.xm * BORA_TILE_CELLS + r.c + 7];
    const float vxp = r.xp < 0 ? 0.f : c.vx[(size_t)r.xp * BORA_TILE_CELLS + r.c];
    beside( vy, yh, 1, r.j == 0, r.j == 7, vym, vyp );
    beside( vz, zh, 8, r.kk == 0, r.kk == 3, vzm, vzp );
    const int EI = g.nx - 1, EJ = g.ny - 1, EK = g.nz - 1;
    const int wall = (float)r.J + 0.5f <= g.voxel_wall + 1.f ? BORA_WALL : BORA_AIR;
    float b[8];
    uint32_t cw[8];
    int count = 0;
#pragma unroll
    for( int q = 0; q < 8; ++q )
    {
        const bool e_i0 = r.i0 + q == 0, e_i1 = r.i0 + q == EI, e_j0 = r.J == 0, e_j1 = r.J == EJ, e_k0 = r.K == 0, e_k1 = r.K == EK;
        const int tt[6] = { e_i0 ? wall : ( q ? flag_of( f.w, q ? q - 1 : 0 ) : f.xm ), e_i1 ? wall : ( q < 7 ? flag_of( f.w, q < 7 ? q + 1 : 7 ) : f.xp ),
                            e_j0 ? wall : flag_of( f.ym, q ), e_j1 ? wall : flag_of( f.yp, q ),
                            e_k0 ? wall : flag_of( f.zm, q ), e_k1 ? wall : flag_of( f.zp, q ) };
        // one axis: the two neighbour values, mirrored at the grid's faces, under the ghost rules
        auto diff = [&]( float v, float lo, float hi, bool e0, bool e1, int t0, int t1 ) {
            const float n0 = e0 ? 2.f * v - hi : lo, n1 = e1 ? 2.f * v - lo : hi;
            const float a = t0 == BORA_AIR ? 2.f * v - n1 : t0 == BORA_WALL ? absr( v ) : n0;
            const float z = t1 == BORA_AIR ? 2.f * v - n0 : t1 == BORA_WALL ? -absr( v ) : n1;
            return ( z - a ) * 0.5f;
        };
        const float dx = diff( vx[q], q ? vx[q ? q - 1 : 0] : vxm, q < 7 ? vx[q < 7 ? q + 1 : 7] : vxp, e_i0, e_i1, tt[0], tt[1] );
        const float dy = diff( vy[q], vym[q], vyp[q], e_j0, e_j1, tt[2], tt[3] );
        const float dz = diff( vz[q], vzm[q], vzp[q], e_k0, e_k1, tt[4], tt[5] );
        const bool fluid = flag_of( f.w, q ) == BORA_FLUID;
        int diag = 6;
        uint32_t mask = 0;
#pragma unroll
        for( int n = 0; n < 6; ++n )
        {
            if( tt[n] == BORA_AIR ) diag += 1;
            else if( tt[n] == BORA_SOLID || tt[n] == BORA_WALL ) diag -= 1;
            else if( tt[n] == BORA_FLUID ) mask |= 1u << n;
        }
        b[q] = fluid ? -( dx + dy + dz ) : 0.f;
        cw[q] = fluid ? BORA_CODE_FLUID | ( (uint32_t)diag << 8 ) | mask : 0u;
        count += fluid ? 1 : 0;
    }
    if( r.mine )
    {
        bora_st8( c.b + r.at(), b );
        *reinterpret_cast<uint4*>( c.code + r.at() ) =
            make_uint4( cw[0] | ( cw[1] << 16 ), cw[2] | ( cw[3] << 16 ), cw[4] | ( cw[5] << 16 ), cw[6] | ( cw[7] << 16 ) );
    }
    count = __reduce_add_sync( 0xffffffffu, count );  // unknowns of the system
    if( ( threadIdx.x & 31 ) == 0 )
    {
        any[threadIdx.x >> 5] = count;
        if( count ) atomicAdd( nfluid, (uint32_t)count );
    }
    __syncthreads();
    if( threadIdx.x < kRowWarps / 2 )
    {
        const int tile = (int)blockIdx.x * ( kRowWarps / 2 ) + (int)threadIdx.x;
        if( tile < ntiles ) tile_fluid[tile] = any[2 * threadIdx.x] || any[2 * threadIdx.x + 1] ? 1 : 0;
    }
}

// ---------------------------------------------------------------------------------
// The solver's tiles (BoraSolveTilesDev): flags -> table.
__global__ void k_tile_fluid( int ntiles, const uint16_t* __restrict__ code, uint8_t* __restrict__ tile_fluid )
{
    for( int s = blockIdx.x * (int)( blockDim.x >> 5 ) + ( threadIdx.x >> 5 ); s < ntiles; s += gridDim.x * (int)( blockDim.x >> 5 ) )
    {
        bool any = false;
        for( int l = threadIdx.x & 31; l < 512; l += 32 ) any = any || ( code[(size_t)s * 512 + l] & BORA_CODE_FLUID );
        any = __any_sync( 0xffffffffu, any );
        if( ( threadIdx.x & 31 ) == 0 ) tile_fluid[s] = any ? 1 : 0;
    }
}

// One CTA: the indices of the flagged (1, not 0) of n items, in order, into out[stride * q + offset],
// and their number; 16 flags per thread and round (a few microseconds for 50 K items).
__global__ void __launch_bounds__( 1024 ) k_flag_list( int n, const uint8_t* __restrict__ flags, int32_t* __restrict__ list,
                                                       int stride, int offset, uint32_t* count, uint32_t* host_count )
{
    __shared__ int wsum[32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    int carry = 0;
    for( int base = 0; base < n; base += 16 * 1024 )
    {
        const int s0 = base + 16 * (int)threadIdx.x;
        uint32_t w[4] = { 0u, 0u, 0u, 0u };
        if( s0 < n )  // the flags are padded to a multiple of 16
        {
            const uint4 f = *reinterpret_cast<const uint4*>( flags + s0 );
            w[0] = f.x; w[1] = f.y; w[2] = f.z; w[3] = f.w;
#pragma unroll
            for( int q = 0; q < 4; ++q )
                for( int b = 0; b < 4; ++b )
                    if( s0 + 4 * q + b >= n ) w[q] &= ~( 0xffu << ( 8 * b ) );
        }
        const int mine = __popc( w[0] ) + __popc( w[1] ) + __popc( w[2] ) + __popc( w[3] );  // flags are 0 or 1
        int inc = mine;
#pragma unroll
        for( int o = 1; o < 32; o <<= 1 )
        {
            const int y = __shfl_up_sync( 0xffffffffu, inc, o );
            if( lane >= o ) inc += y;
        }
        if( lane == 31 ) wsum[wid] = inc;
        __syncthreads();
        if( wid == 0 )
        {
            int v = wsum[lane];
#pragma unroll
            for( int o = 1; o < 32; o <<= 1 )
            {
                const int y = __shfl_up_sync( 0xffffffffu, v, o );
                if( lane >= o ) v += y;
            }
            wsum[lane] = v;
        }
        __syncthreads();
        int out = carry + inc - mine + ( wid ? wsum[wid - 1] : 0 );
        for( int b = 0; b < 16; ++b )
            if( ( w[b >> 2] >> ( 8 * ( b & 3 ) ) ) & 1u ) list[stride * (size_t)out++ + offset] = s0 + b;
        carry += wsum[31];
        __syncthreads();  // wsum is rewritten next
    }
    if( threadIdx.x == 0 )
    {
        *count = (uint32_t)carry;
        *(volatile uint32_t*)host_count = (uint32_t)carry;
    }
}

// The face neighbours of the solver's tiles (-1: not a solver tile), eight threads per tile.
__global__ void k_solve_nbrs( const uint32_t* __restrict__ count, const int32_t* __restrict__ nbr,
                              const uint8_t* __restrict__ tile_fluid, int32_t* __restrict__ tab )
{
    const size_t total = (size_t)*count * 8;
    for( size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x; q < total; q += (size_t)gridDim.x * blockDim.x )
    {
        const int f = (int)( q & 7 );
        if( f == 7 ) tab[q] = 0;
        if( f >= 6 ) continue;
        const int sg = ( f & 1 ) ? 1 : -1;
        const int ns = nbr[(size_t)tab[( q & ~(size_t)7 ) + 6] * 27 + bora_dir( f < 2 ? sg : 0, f == 2 || f == 3 ? sg : 0, f >= 4 ? sg : 0 )];
        tab[q] = ns >= 0 && tile_fluid[ns] ? ns : -1;
    }
}

__device__ __forceinline__ int solve_slot( const int4* tab, int t ) { return __ldg( &tab[2 * (size_t)t + 1].z ); }

// ---------------------------------------------------------------------------------
// Wavefront tables of an 8^3 tile: cells ordered by plane i+j+k (0..21). Kept in global
// memory and copied to shared memory by every CTA that sweeps planes (lanes of a warp
// read different entries, which a constant-memory table would serialise).
__device__ uint16_t g_plane_cells[512];
__device__ uint16_t g_plane_start[23];

struct PlaneTables
{
    uint16_t cells[512];
    uint16_t start[23];
    PlaneTables()
    {
        int n = 0;
        for( int s = 0; s <= 21; ++s )
        {
            start[s] = (uint16_t)n;
            for( int l = 0; l < 512; ++l )
            {
                const int i = l & 7, j = ( l >> 3 ) & 7, k = l >> 6;
                if( i + j + k == s ) cells[n++] = (uint16_t)l;
            }
        }
        start[22] = (uint16_t)n;
    }
};

void ensure_tables()
{
    static BoraPerDevice ready;
    ready.get( [] {
        static const PlaneTables tbl;
        cudaMemcpyToSymbol( g_plane_cells, tbl.cells, sizeof( tbl.cells ) );
        cudaMemcpyToSymbol( g_plane_start, tbl.start, sizeof( tbl.start ) );
        cudaDeviceSynchronize();  // the tables are in place before any stream's kernel reads them
        return 1;
    } );
}

int num_sms()
{
    static BoraPerDevice sms;
    return sms.get( [] {
        int dev = 0, n = 0;
        cudaGetDevice( &dev );
        cudaDeviceGetAttribute( &n, cudaDevAttrMultiProcessorCount, dev );
        return n > 0 ? n : 152;
    } );
}

__device__ inline void load_plane_tables( uint16_t* pc, uint16_t* ps )
{
    for( int q = threadIdx.x; q < 512; q += blockDim.x ) pc[q] = g_plane_cells[q];
    if( threadIdx.x < 23 ) ps[threadIdx.x] = g_plane_start[threadIdx.x];
}

__device__ inline int code_diag( uint16_t c ) { return ( c >> 8 ) & 15; }

// Block-MIC(0) pivots (MIC(0) of BLAS.cu:211-262 with tau = 0.97, restricted to the
// couplings inside each 8^3 tile so that tiles factor independently), stored squared and
// rotated (mic_sweeps). One warp per tile, persistent over tiles.
constexpr int kTilesPerCta = 4;

__global__ void __launch_bounds__( 32 * kTilesPerCta ) k_mic_factor( BoraSolveTilesDev ft,
                                                                     const uint16_t* __restrict__ code,
                                                                     float* __restrict__ minv )
{
    __shared__ float sm[kTilesPerCta][512];
    __shared__ uint16_t sc[kTilesPerCta][512];
    __shared__ uint16_t pc[512], ps[23];
    load_plane_tables( pc, ps );
    __syncthreads();
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const float tau = 0.97f;
    const int nft = (int)*ft.count;
    for( int t = blockIdx.x * kTilesPerCta + w; t < nft; t += gridDim.x * kTilesPerCta )
    {
        const size_t base = (size_t)solve_slot( ft.tab, t ) * 512;
        for( int l = lane; l < 512; l += 32 ) { sc[w][l] = code[base + l]; sm[w][l] = 0.f; }
        __syncwarp();
        for( int p = 0; p <= 21; ++p )
        {
            for( int q = ps[p] + lane; q < ps[p + 1]; q += 32 )
            {
                const int l = pc[q];
                const uint16_t cc = sc[w][l];
                if( !( cc & BORA_CODE_FLUID ) ) continue;
                const int li = l & 7, lj = ( l >> 3 ) & 7, lk = l >> 6;
                const float diag = (float)code_diag( cc );
                float e = diag, e2 = 0.f;
                if( li > 0 && ( cc & 1u ) )
                {
                    const int m = l - 1;
                    const uint16_t cm = sc[w][m];
                    const float M = sm[w][m];
                    const float a = ( lj < 7 && ( cm & 8u ) ) ? 1.f : 0.f;    // m+y inside the tile and fluid
                    const float b = ( lk < 7 && ( cm & 32u ) ) ? 1.f : 0.f;   // m+z
                    e -= M * M;
                    e2 += ( a + b ) * ( M * M );
                }
                if( lj > 0 && ( cc & 4u ) )
                {
                    const int m = l - 8;
                    const uint16_t cm = sc[w][m];
                    const float M = sm[w][m];
                    const float a = ( li < 7 && ( cm & 2u ) ) ? 1.f : 0.f;    // m+x
                    const float b = ( lk < 7 && ( cm & 32u ) ) ? 1.f : 0.f;   // m+z
                    e -= M * M;
                    e2 += ( a + b ) * ( M * M );
                }
                if( lk > 0 && ( cc & 16u ) )
                {
                    const int m = l - 64;
                    const uint16_t cm = sc[w][m];
                    const float M = sm[w][m];
                    const float a = ( li < 7 && ( cm & 2u ) ) ? 1.f : 0.f;    // m+x
                    const float b = ( lj < 7 && ( cm & 8u ) ) ? 1.f : 0.f;    // m+y
                    e -= M * M;
                    e2 += ( a + b ) * ( M * M );
                }
                e -= tau * e2;
                if( e < diag * 0.25f ) e = diag;
                sm[w][l] = 1.f / sqrtf( e + 1e-30f );
            }
            __syncwarp();
        }
        // squared, each row rotated as mic_sweeps reads it
        for( int l = lane; l < 512; l += 32 )
            minv[base + ( l & ~7 ) + ( ( l + ( l >> 3 & 7 ) + ( l >> 6 ) + 1 ) & 7 )] = sm[w][l] * sm[w][l];
        __syncwarp();
    }
}

// ---------------------------------------------------------------------------------
// PCG update: r -= alpha q; z = M^-1 r (block-MIC(0) forward and backward sweeps over the
// tile's 22 wavefront planes i+j+k = p); rz = r.z and rr = r.r, FP64-accurate. The matching
// e += alpha d is applied by the next direction kernel (which reads d anyway) or by the
// refinement step. One warp per tile, persistent over tiles (every warp gets the same number
// of tiles).
//
// The sweeps run in registers. Each lane owns two x-rows of the tile that are neighbours in z,
// row A = (j, k = 2 kq) and row B = (j, k + 1), j = lane & 7, kq = lane >> 3. Step u of a sweep
// handles cell i = u - (j + k) - 1 of every row at once. In the scaled unknowns w = M y and the
// squared pivots M2 = M^2 (which k_mic_factor stores) the sweeps are
//   forward   w = M2 t, t = r + (w_-x + w_-y + w_-z)
//   backward  z = w + M2 (z_+x + z_+y + z_+z),
// so a step needs its neighbours' single values of the step before: -x and the z neighbour
// inside the pair are the lane's own registers, the other y and z neighbours are three
// shuffles. A row's cells sit in eight registers rotated by (j + k + 1) mod 8, so that step u
// finds its cell in register u mod 8 in every lane (r is rotated in three select stages; M2 is
// stored rotated). Steps outside a row's eight cells yield 0, which feeds the row's first cell a
// zero neighbour. r.z = sum of w t (r.M^-1 r = y.y), all terms >= 0, in FP32 over four cells (a
// row's eight lie at consecutive steps, so exactly four of them at steps with bit 2 set), then in
// double-float. Non-fluid cells have M2 = 0 and r = 0.
//
// Bound by latency and issue: 44 dependent steps of a shuffle and three arithmetic
// instructions, about 900 warp instructions per tile. With the tile in shared memory (11 shared
// accesses per row and step pair, 78 % of the shared pipe) a launch took 32.5 us at 256^3 (7926 tiles)
// with an event on either side, in registers 22 (3.7 TB/s of its 20 B per cell), and 18 over the
// solver's tiles alone; 8.4 against 11.9 us at 64^3 (240 tiles). 16 warps per SM without spills beat 20 .. 32 with
// (23.3 against 23.5 .. 26.1 ms per 256^3 step), and loading the next tile during the sweeps
// gains nothing (23.3 .. 24.3 ms).
constexpr int kUpdWarps = 4;

// v[i] -> v[(i + rho) mod 8]
__device__ __forceinline__ void rotate8( float* v, int rho )
{
#pragma unroll
    for( int b = 1; b < 8; b <<= 1 )
    {
        float t[8];
        const bool on = ( rho & b ) != 0;
#pragma unroll
        for( int i = 0; i < 8; ++i ) t[i] = on ? v[( i - b ) & 7] : v[i];
#pragma unroll
        for( int i = 0; i < 8; ++i ) v[i] = t[i];
    }
}

// z = M^-1 r of one tile: rA, rB hold the lane's rows of r and return z (both in cell order);
// mA, mB the rows' squared pivots as stored (rotated). Adds the lane's part of r.z to prz. ROLLED: a
// third of the code, for a kernel whose one warp per SM partition would wait for its instructions
// (the grid kernel is faster unrolled: 18.3 against 18.7 ms of GPU time per 256^3 step).
template <bool ROLLED>
__device__ __forceinline__ void mic_sweeps( float* rA, float* rB, const float* mA, const float* mB, DF& prz )
{
    constexpr unsigned kAllLanes = 0xffffffffu;
    const int lane = threadIdx.x & 31, j = lane & 7, kq = lane >> 3, sA = j + 2 * kq, rho = ( sA + 1 ) & 7;
    const float ym = j > 0 ? 1.f : 0.f, yp = j < 7 ? 1.f : 0.f, zm = kq > 0 ? 1.f : 0.f, zp = kq < 3 ? 1.f : 0.f;
    const unsigned live = 0xffu << ( sA + 1 );  // bit u: row A has a cell at step u (row B: at step u + 1)
    rotate8( rA, rho );
    rotate8( rB, rho );  // row B's cell of step u is register (u - 1) mod 8
    float wA = 0.f, wB = 0.f, rzA[2] = { 0.f, 0.f }, rzB[2] = { 0.f, 0.f };
    // three rounds of eight steps (none past step 22): a register's steps are eight apart, so the
    // round can be the body of a loop
    constexpr int kRounds = ROLLED ? 1 : 3;
#pragma unroll kRounds
    for( int round = 0; round < 3; ++round )
    {
        const unsigned lv = live >> ( 8 * round );  // bit v: row A has a cell at step v of the round
#pragma unroll
        for( int v = 1; v <= 8; ++v )
        {
            if( !ROLLED && 8 * round + v > 22 ) continue;
            const bool a = ( lv >> v ) & 1u, b = ( lv >> ( v - 1 ) ) & 1u;
            const float yA = __shfl_up_sync( kAllLanes, wA, 1 ), yB = __shfl_up_sync( kAllLanes, wB, 1 );
            const float zA = __shfl_up_sync( kAllLanes, wB, 8 );
            float& cA = rA[v & 7];
            float& cB = rB[v - 1];
            const float tA = fmaf( zm, zA, fmaf( ym, yA, cA + wA ) );
            const float tB = fmaf( ym, yB, ( cB + wB ) + wA );
            wA = a ? mA[v & 7] * tA : 0.f;
            wB = b ? mB[v & 7] * tB : 0.f;
            rzA[( v >> 2 ) & 1] = fmaf( wA, tA, rzA[( v >> 2 ) & 1] );
            rzB[( v >> 2 ) & 1] = fmaf( wB, tB, rzB[( v >> 2 ) & 1] );
            cA = a ? wA : cA;
            cB = b ? wB : cB;
        }
    }
    float zA = 0.f, zB = 0.f;
#pragma unroll kRounds
    for( int round = 2; round >= 0; --round )
    {
        const unsigned lv = live >> ( 8 * round );
#pragma unroll
        for( int v = 8; v >= 1; --v )
        {
            if( !ROLLED && 8 * round + v > 22 ) continue;
            const bool a = ( lv >> v ) & 1u, b = ( lv >> ( v - 1 ) ) & 1u;
            const float yA = __shfl_down_sync( kAllLanes, zA, 1 ), yB = __shfl_down_sync( kAllLanes, zB, 1 );
            const float nB = __shfl_down_sync( kAllLanes, zA, 8 );
            float& cA = rA[v & 7];
            float& cB = rB[v - 1];
            const float sumA = fmaf( yp, yA, zA + zB ), sumB = fmaf( zp, nB, fmaf( yp, yB, zB ) );
            zA = a ? fmaf( mA[v & 7], sumA, cA ) : 0.f;
            zB = b ? fmaf( mB[v & 7], sumB, cB ) : 0.f;
            cA = a ? zA : cA;
            cB = b ? zB : cB;
        }
    }
    rotate8( rA, ( 8 - rho ) & 7 );
    rotate8( rB, ( 8 - rho ) & 7 );
#pragma unroll
    for( int q = 0; q < 2; ++q ) prz = df_add_f( df_add_f( prz, rzA[q] ), rzB[q] );
}

// The update of the warp's tiles first, first + tstride, ...: r -= alpha q, z = M^-1 r; r.z and
// r.r accumulated into prz, prr. alpha_of() is called once, by every thread of the block, after
// the first tile's loads have been issued.
template <class AlphaOf>
__device__ __forceinline__ void pcg_update_tiles( const BoraSolveTilesDev& ft, const BoraSolverDev& sv, AlphaOf alpha_of, unsigned bid,
                                                  unsigned G, DF& prz, DF& prr )
{
    // the tiles' slots, read a tile ahead (no kernel of the chain writes the table)
    const int tstride = (int)G * kUpdWarps, first = (int)bid * kUpdWarps + ( threadIdx.x >> 5 );
    int next = first < ft.n ? solve_slot( ft.tab, first ) : 0;
    const int lane = threadIdx.x & 31;
    const size_t row = 8 * (size_t)( ( lane & 7 ) + 16 * ( lane >> 3 ) );  // row A; row B follows 64 cells on
    float rA[8], rB[8], qA[8], qB[8], mA[8], mB[8];
    auto load_tile = [&]( int s ) {
        const size_t o = (size_t)s * 512 + row;
        bora_ld8( sv.r + o, rA ); bora_ld8( sv.r + o + 64, rB );
        bora_ld8( sv.q + o, qA ); bora_ld8( sv.q + o + 64, qB );
    };
    bora_pdl_wait();  // the previous kernel's results are complete from here
    if( first < ft.n ) load_tile( next );
    const float alpha = alpha_of();
    for( int t = first; t < ft.n; t += tstride )
    {
        const int s = next;
        const size_t o = (size_t)s * 512 + row;
        if( t != first ) load_tile( s );
        if( t + tstride < ft.n ) next = solve_slot( ft.tab, t + tstride );
        bora_ld8( sv.minv + o, mA );  // not with the first loads: the registers they take there cost more (spills)
        bora_ld8( sv.minv + o + 64, mB );
#pragma unroll
        for( int i = 0; i < 8; ++i )
        {
            rA[i] = fmaf( -alpha, qA[i], rA[i] );
            rB[i] = fmaf( -alpha, qB[i], rB[i] );
        }
        bora_st8( sv.r + o, rA );
        bora_st8( sv.r + o + 64, rB );
#pragma unroll
        for( int h = 0; h < 8; h += 4 )
        {
            prr = df_add_f( prr, dot4( make_float4( rA[h], rA[h + 1], rA[h + 2], rA[h + 3] ), make_float4( rA[h], rA[h + 1], rA[h + 2], rA[h + 3] ) ) );
            prr = df_add_f( prr, dot4( make_float4( rB[h], rB[h + 1], rB[h + 2], rB[h + 3] ), make_float4( rB[h], rB[h + 1], rB[h + 2], rB[h + 3] ) ) );
        }
        mic_sweeps<false>( rA, rB, mA, mB, prz );
        bora_st8( sv.z + o, rA );
        bora_st8( sv.z + o + 64, rB );
    }
}

__global__ void __launch_bounds__( 32 * kUpdWarps, 4 ) k_pcg_update( BoraSolveTilesDev ft, BoraSolverDev sv,
                                                                  BoraReduceDev red, int ndq, int slot_rz_in,
                                                                  int slot_dq_in )
{
    __shared__ float2 s_dq[kUpdWarps];
    bora_pdl_trigger();
    DF prz{ 0.f, 0.f }, prr{ 0.f, 0.f };
    auto alpha_of = [&]() -> float {
        if( slot_rz_in < 0 ) return 0.f;
        const DF dq = part_collect( red.part_dq, ndq, s_dq );
        if( blockIdx.x == 0 && threadIdx.x == 0 ) ring_store( red, slot_dq_in, dq, false );
        return df_ratio( red.ringf[slot_rz_in], make_float2( dq.hi, dq.lo ) );
    };
    if( ft.n > 0 ) pcg_update_tiles( ft, sv, alpha_of, blockIdx.x, gridDim.x, prz, prr );
    part_publish( prz, prr, red.part_rz, red.part_rr, blockIdx.x );
}

// ---------------------------------------------------------------------------------
// PCG direction: e += alpha d (the previous update's step, pending); d' = z + beta d;
// q = A d'; dq = d'.q (d double-buffered). One warp per half tile (the z-layers 0..3 or 4..7),
// persistent over half tiles; a lane owns one x-row (lane = j + 8 (k mod 4)), read and written as
// 32-byte vectors. The stencil's x neighbours are the lane's own registers, its y and z neighbours
// inside the half come from other lanes by shuffles, and the rows across the half's faces (the
// other half, the face-neighbour tiles) are loaded by the lanes that need them (d' formed the same
// way; an inactive neighbour tile contributes 0). Non-fluid cells hold d = z = 0, so the stencil
// sum runs over all six neighbours in the fixed order -x, +x, -y, +y, -z, +z; the dot product adds
// d'.q of two x-neighbour cells in float, then into a double-float sum.
//
// Waits on its loads (long scoreboard), so it wants warps in flight and few sectors per load: a
// lane with two rows needs 122 registers for the same loads in flight (31.2 us per launch with
// 16-byte loads at 72 registers, 256^3, an event on either side; 26.8 us so, 20.6 over the solver's tiles alone).
constexpr int kDirWarps = 4;

// The direction step of the warp's half tiles bid * kDirWarps + warp, then every G * kDirWarps:
// returns the thread's d'.q. coef(): the pair (beta, alpha of the pending e += alpha d), called
// once by every thread of the block after the first half tile's loads have been issued; upd_e:
// that update is pending.
template <class Coef>
__device__ __forceinline__ DF pcg_direction_tiles( const BoraSolveTilesDev& ft, const uint16_t* __restrict__ code,
                                                   const BoraSolverDev& sv, int dsel_in, Coef coef, bool upd_e, unsigned bid,
                                                   unsigned G )
{
    const float* dold = dsel_in ? sv.d[1] : sv.d[0];  // selects keep sv out of local memory
    float* dnew = dsel_in ? sv.d[0] : sv.d[1];
    const int lane = threadIdx.x & 31, j = lane & 7, kk = lane >> 3;
    constexpr unsigned kAll = 0xffffffffu;
    DF pdq{ 0.f, 0.f };
    float beta = 0.f, alpha = 0.f;
    float d[8] = {}, z[8] = {};
    const int nh = 2 * ft.n, stride = (int)G * kDirWarps;
    const int first = min( (int)bid * kDirWarps + (int)( threadIdx.x >> 5 ), nh - 1 );
    // a half tile's slot, read one ahead (no kernel of the chain writes the table)
    int next = solve_slot( ft.tab, first >> 1 );
    auto load_rows = [&]( size_t g, bool mine ) {
        if( !mine ) return;
        bora_ld8( dold + g, d );
        bora_ld8( sv.z + g, z );
    };
    bora_pdl_wait();  // the previous kernel's results (ring, partial sums, z, d, e) are complete from here
    load_rows( (size_t)next * 512 + ( first & 1 ) * 256 + 8 * lane, (int)bid * kDirWarps + (int)( threadIdx.x >> 5 ) < nh );
    {
        const float2 c = coef();
        beta = c.x;
        alpha = c.y;
    }
    // (a bound of the block's, as in the update; a warp past the last half tile stores nothing)
#pragma unroll 1
    for( int base = (int)bid * kDirWarps; base < nh; base += stride )
    {
        const int h0 = base + (int)( threadIdx.x >> 5 ), h = min( h0, nh - 1 );
        const bool mine = h0 < nh;
        const int s = next, hi = h & 1;
        const int cA = hi * 256 + 8 * lane;
        const size_t g = (size_t)s * 512 + cA;
        const int4 n0 = __ldg( ft.tab + 2 * (size_t)( h >> 1 ) ), n1 = __ldg( ft.tab + 2 * (size_t)( h >> 1 ) + 1 );
        const int smx = n0.x, spx = n0.y, smy = n0.z, spy = n0.w, sz = hi ? n1.y : n1.x;
        const int hn = min( h0 + stride, nh - 1 );
        next = solve_slot( ft.tab, hn >> 1 );
        const uint4 w = *reinterpret_cast<const uint4*>( code + g );
        float e[8];
        if( upd_e ) bora_ld8( sv.e + g, e );
        auto halo1 = [&]( int t, int c ) { return t < 0 ? 0.f : fmaf( beta, dold[(size_t)t * 512 + c], sv.z[(size_t)t * 512 + c] ); };
        auto halo8 = [&]( int t, int c, float* v ) {
            if( t < 0 ) { for( int i = 0; i < 8; ++i ) v[i] = 0.f; return; }
            float dd[8];
            bora_ld8( dold + (size_t)t * 512 + c, dd );
            bora_ld8( sv.z + (size_t)t * 512 + c, v );
#pragma unroll
            for( int i = 0; i < 8; ++i ) v[i] = fmaf( beta, dd[i], v[i] );
        };
        const float xm = halo1( smx, cA + 7 ), xp = halo1( spx, cA );
        const int yt = j == 0 ? smy : ( j == 7 ? spy : -1 ), yc = cA + ( j == 0 ? 56 : -56 );
        // the z neighbour rows outside the warp's half: the other half, or the neighbour tile
        const int zt = kk == 0 ? ( hi ? s : sz ) : ( kk == 3 ? ( hi ? sz : s ) : -1 );
        const int zc = 8 * j + ( kk == 0 ? ( hi ? 192 : 448 ) : ( hi ? 0 : 256 ) );
        float yh[8], zh[8], q[8];
        halo8( yt, yc, yh );
        halo8( zt, zc, zh );
        if( upd_e )
        {
#pragma unroll
            for( int i = 0; i < 8; ++i ) e[i] = fmaf( alpha, d[i], e[i] );
            if( mine ) bora_st8( sv.e + g, e );
        }
#pragma unroll
        for( int i = 0; i < 8; ++i ) d[i] = fmaf( beta, d[i], z[i] );
        if( mine ) bora_st8( dnew + g, d );
        const uint32_t cw[4] = { w.x, w.y, w.z, w.w };
#pragma unroll
        for( int i = 0; i < 8; ++i )
        {
            float ym = __shfl_up_sync( kAll, d[i], 1 ), yp = __shfl_down_sync( kAll, d[i], 1 );
            if( j == 0 ) ym = yh[i];
            if( j == 7 ) yp = yh[i];
            float zm = __shfl_up_sync( kAll, d[i], 8 ), zp = __shfl_down_sync( kAll, d[i], 8 );
            if( kk == 0 ) zm = zh[i];
            if( kk == 3 ) zp = zh[i];
            const uint32_t c = i & 1 ? cw[i >> 1] >> 16 : cw[i >> 1] & 0xffffu;
            q[i] = 0.f;
            if( c & BORA_CODE_FLUID )
            {
                float acc = 0.f;
                acc += i > 0 ? d[i > 0 ? i - 1 : 0] : xm; acc += i < 7 ? d[i < 7 ? i + 1 : 7] : xp;
                acc += ym; acc += yp; acc += zm; acc += zp;
                q[i] = fmaf( (float)code_diag( (uint16_t)c ), d[i], -acc );
            }
        }
        if( mine )
        {
#pragma unroll
            for( int i = 0; i < 8; i += 2 ) pdq = df_add_f( pdq, fmaf( d[i + 1], q[i + 1], d[i] * q[i] ) );
            bora_st8( sv.q + g, q );
        }
        load_rows( (size_t)next * 512 + ( hn & 1 ) * 256 + 8 * lane, h0 + stride < nh );
    }
    return pdq;
}

__device__ __forceinline__ void pcg_direction_body( const BoraSolveTilesDev& ft, const uint16_t* __restrict__ code,
                                                    const BoraSolverDev& sv, int dsel_in, const BoraReduceDev& red, int nparts, int slot_rz_new, int slot_rr,
                                                    int slot_rz_old, int slot_a_rz, int slot_a_dq, bool host_rr, unsigned bid,
                                                    unsigned G )
{
    __shared__ float2 s_rz[kDirWarps], s_rr[kDirWarps];
    bora_pdl_trigger();
    auto coef = [&]() -> float2 {
        const DF rz = part_collect( red.part_rz, nparts, s_rz );
        if( bid == G - 1 )  // the last block (never the one with more tiles) finishes rr for the host
        {
            const DF rr = part_collect( red.part_rr, nparts, s_rr );
            if( threadIdx.x == 0 )
            {
                ring_store( red, slot_rz_new, rz, false );
                ring_store( red, slot_rr, rr, host_rr );
            }
        }
        return make_float2( slot_rz_old < 0 ? 0.f : df_ratio( make_float2( rz.hi, rz.lo ), red.ringf[slot_rz_old] ),
                            slot_a_rz < 0 ? 0.f : df_ratio( red.ringf[slot_a_rz], red.ringf[slot_a_dq] ) );
    };
    const DF pdq = pcg_direction_tiles( ft, code, sv, dsel_in, coef, slot_a_rz >= 0, bid, G );
    part_publish( pdq, DF{ 0.f, 0.f }, red.part_dq, nullptr, bid );
}

__global__ void __launch_bounds__( 32 * kDirWarps, 6 ) k_pcg_direction( BoraSolveTilesDev ft,
                                                                    const uint16_t* __restrict__ code, BoraSolverDev sv,
                                                                    int dsel_in, BoraReduceDev red, int nparts,
                                                                    int slot_rz_new, int slot_rr, int slot_rz_old,
                                                                    int slot_a_rz, int slot_a_dq, bool host_rr )
{
    pcg_direction_body( ft, code, sv, dsel_in, red, nparts, slot_rz_new, slot_rr, slot_rz_old, slot_a_rz, slot_a_dq,
                        host_rr, blockIdx.x, gridDim.x );
}

// Batched: each simulation on its own grid of m.grid[kGridDir] blocks.
__global__ void __launch_bounds__( 32 * kDirWarps ) k_pcg_direction_batch( const __grid_constant__ BoraBatchLaunch L )
{
    unsigned bid;
    const int k = bora_batch_member( L, blockIdx.x, &bid );
    const BoraMemberSolve& m = L.ms[k];
    const BoraMemberSlots& q = L.sl[k];
    pcg_direction_body( m.ft, m.code, m.sv, q.dsel, m.red, m.grid[kGridPass0R], q.rz_new, q.rr_new, q.rz_old,
                        q.a_rz, q.a_dq, q.chk != 0, bid, (unsigned)m.grid[kGridDir] );
}

// ---------------------------------------------------------------------------------
// Persistent plain PCG: one cooperative launch runs a refinement pass's inner iterations -
// the first update (z = M^-1 r), then direction and update per iteration - with a grid-wide
// barrier after each phase instead of a kernel boundary. The phases are the kernels' own tile
// loops; a phase's sums are formed per block (warps in a fixed order), stored, and after the
// barrier every block adds all blocks' values in the same fixed order, so each block holds
// the same bits without a second barrier. The pass stops after the update whose ||r|| reaches
// the target (checked in the kernel, the same in every block) or after max_inner iterations.
//
// Every barrier wait is bounded: a block that has spun `limit` times, or that sees another
// block's error, sets BORA_REDUCE_ERR_BARRIER in the error word and returns; every other block
// then runs out of its own waits and returns too, and the host reports BORA_ERR_INTERNAL.
struct PcgPersistArgs
{
    BoraSolveTilesDev ft;
    const uint16_t* code;
    BoraSolverDev sv;
    BoraReduceDev red;
    int dsel;                  // the current search-direction buffer
    int slot_rz_prev;          // r.z before the last update of the previous pass, or -1 (restart)
    int max_inner;
    double target;             // stop once ||r|| <= target
    int slot_a_rz, slot_a_dq;  // out: the last update's alpha = a_rz / a_dq (its e += alpha d is pending);
                               // the last r.r is left as the one partial sum part_rr[0]
    uint32_t* iters;           // out: iterations run
    unsigned* bar;             // barrier count and generation (zeroed before the launch)
    unsigned expect;           // blocks a barrier waits for (gridDim.x)
    unsigned limit;            // spins per barrier wait
    double* part;              // 3 * gridDim.x block sums
};

__device__ __forceinline__ bool grid_barrier( const PcgPersistArgs& a )
{
    __shared__ int s_ok;
    __syncthreads();
    if( threadIdx.x == 0 )
    {
        volatile unsigned* gen = a.bar + 1;
        volatile uint32_t* err = a.red.err;
        int ok = 1;
        const unsigned g = *gen;
        __threadfence();
        if( atomicAdd( a.bar, 1u ) == a.expect - 1 )
        {
            atomicExch( a.bar, 0u );
            __threadfence();
            atomicAdd( a.bar + 1, 1u );
        }
        else
        {
            for( unsigned n = 0; *gen == g; ++n )
            {
                if( n >= a.limit || *err )
                {
                    atomicOr( a.red.err, (uint32_t)BORA_REDUCE_ERR_BARRIER );
                    ok = 0;
                    break;
                }
                __nanosleep( 128 );
            }
        }
        __threadfence();
        s_ok = ok;
    }
    __syncthreads();
    return s_ok != 0;
}

// The block's total of v (valid in every lane of every warp), stored at part[blockIdx.x].
__device__ __forceinline__ void block_sum_store( double v, double* part )
{
    __shared__ double w[32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    if( lane == 0 ) w[wid] = v;
    __syncthreads();
    if( threadIdx.x == 0 )
    {
        double t = 0.0;
        for( int q = 0; q < nw; ++q ) t += w[q];
        part[blockIdx.x] = t;
    }
    __syncthreads();  // w is reused by the next call
}

// The sum of part[0 .. nb) in a fixed order (the first warp: lane-strided, then a fixed
// shuffle tree), returned in every thread.
__device__ __forceinline__ double grid_sum( const double* part, unsigned nb )
{
    __shared__ double s_total;
    if( threadIdx.x < 32 )
    {
        double t = 0.0;
        for( unsigned q = threadIdx.x; q < nb; q += 32 ) t += __ldcg( part + q );
        t = warp_sum( t );
        if( threadIdx.x == 0 ) s_total = t;
    }
    __syncthreads();
    const double v = s_total;
    __syncthreads();
    return v;
}

__global__ void __launch_bounds__( 32 * kUpdWarps, 3 ) k_pcg_persistent( const __grid_constant__ PcgPersistArgs a )
{
    static_assert( kUpdWarps == kDirWarps, "one block shape for both phases" );
    const unsigned G = gridDim.x;
    double* const pd = a.part;                // d'.q
    double* const pz = a.part + G;            // r.z
    double* const pr = a.part + 2 * (size_t)G;  // r.r
    double rz_prev = a.slot_rz_prev >= 0 ? a.red.ring[a.slot_rz_prev] : -1.0;
    // the pass's first update: z = M^-1 r (alpha 0)
    DF prz{ 0.f, 0.f }, prr{ 0.f, 0.f };
    pcg_update_tiles( a.ft, a.sv, [] { return 0.f; }, blockIdx.x, G, prz, prr );
    block_sum_store( df_warp_sum( prz ), pz );
    block_sum_store( df_warp_sum( prr ), pr );
    if( !grid_barrier( a ) ) return;
    double rz = grid_sum( pz, G ), rr = grid_sum( pr, G );
    double a_rz = -1.0, a_dq = 1.0;
    int dsel = a.dsel, it = 0;
    while( it < a.max_inner )
    {
        const float beta = rz_prev < 0.0 ? 0.f : (float)( rz / rz_prev );
        const float alpha_e = a_rz < 0.0 ? 0.f : (float)( a_rz / a_dq );
        const DF pdq = pcg_direction_tiles( a.ft, a.code, a.sv, dsel, [=] { return make_float2( beta, alpha_e ); },
                                            a_rz >= 0.0, blockIdx.x, G );
        block_sum_store( df_warp_sum( pdq ), pd );
        if( !grid_barrier( a ) ) return;
        const double dq = grid_sum( pd, G );
        dsel ^= 1;
        prz = DF{ 0.f, 0.f };
        prr = DF{ 0.f, 0.f };
        const float alpha = (float)( rz / dq );
        pcg_update_tiles( a.ft, a.sv, [=] { return alpha; }, blockIdx.x, G, prz, prr );
        block_sum_store( df_warp_sum( prz ), pz );
        block_sum_store( df_warp_sum( prr ), pr );
        if( !grid_barrier( a ) ) return;
        a_rz = rz;
        a_dq = dq;
        rz_prev = rz;
        rz = grid_sum( pz, G );
        rr = grid_sum( pr, G );
        ++it;
        if( !( rr > 0.0 ) || sqrt( rr ) <= a.target ) break;
    }
    if( blockIdx.x == 0 && threadIdx.x == 0 )
    {
        auto pair = []( double v ) { return DF{ (float)v, (float)( v - (double)(float)v ) }; };
        ring_store( a.red, a.slot_a_rz, pair( a_rz ), false );
        ring_store( a.red, a.slot_a_dq, pair( a_dq ), false );
        a.red.part_rr[0] = make_float2( pair( rr ).hi, pair( rr ).lo );  // finished by the refinement
        *a.iters = (uint32_t)it;
    }
}

// ---------------------------------------------------------------------------------
// Resident plain PCG: a refinement pass's inner iterations in one cooperative launch for systems
// whose tiles fit one warp each, every vector of a tile in its warp's registers. Per iteration the
// blocks meet twice:
//   direction  d = z + beta d, q = A d; d.q
//   update     e += alpha d, r -= alpha q, z = M^-1 r (mic_sweeps); r.z, r.r; z stored
// Only z crosses tiles through memory: a lane that needs a neighbour tile's cells keeps their d
// as well and forms d = z + beta d for them itself. The stop test runs on the device.
//
// A meeting is a sum: a block stores its partial sums as 64-bit words of a float and a tag (the
// meeting's number), and every block's first warp polls all blocks' words, so a value is its own
// arrival signal - no counter, no second read. A tag is never reused while a word can hold it
// (the host hands each launch its own range). z is stored before the block's fence and words, and
// read past L1 after the poller's fence. Each wait is bounded: a warp that polls `limit` times, or
// sees another block's error, sets BORA_REDUCE_ERR_BARRIER and its block returns; the other blocks
// then run out in turn, and the host finds no iteration count.
//
// Bound by latency. Of 10.7 K cycles per iteration at 15 tiles the sweeps and sums take 2.7 K, the
// fence 1.0 K, the two meetings 4.6 K, the stencil 1.2 K. Code that fits the instruction caches
// matters (one warp per SM partition hides no fetch: 10 x slower at 100 KB): rolled sweeps, one
// copy of each part, control flow that the compiler knows to be uniform.
struct PcgResidentArgs
{
    BoraSolveTilesDev ft;
    const uint16_t* code;
    BoraSolverDev sv;
    BoraReduceDev red;
    int dsel;               // the buffer of the last search direction (read and left there)
    int slot_rz_prev;       // r.z before the last update of the previous pass, or -1 (restart)
    int max_inner;
    int check, beyond;      // iterations between stop tests; iterations that a pass runs on after one that holds
    double target2;         // stop once r.r <= target2
    float above;            // an r.r that is not: its FP64 test, 0.2 us (0.8 with a root), is only formed at the end
    int slot_a_rz;          // out: r.z before the last update; r.r is left as the one partial sum part_rr[0]
    uint32_t* iters;        // out (mapped host memory): iterations run; not written when a wait ran out
    ulonglong2* words_rz;   // two per block: r.z, r.r
    ulonglong2* words_dq;   // one per block
    uint32_t tag;           // first tag of the launch
    unsigned expect;        // blocks a meeting waits for (gridDim.x)
    unsigned limit;         // polls per wait
};

__device__ __forceinline__ ulonglong2 tagged( DF v, uint32_t tag )
{
    const unsigned long long t = (unsigned long long)tag << 32;
    return make_ulonglong2( t | __float_as_uint( v.hi ), t | __float_as_uint( v.lo ) );
}

__device__ __forceinline__ void store_words( ulonglong2* p, ulonglong2 v )
{
    asm volatile( "st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"( p ), "l"( v.x ), "l"( v.y ) : "memory" );
}

__device__ __forceinline__ ulonglong2 load_words( const ulonglong2* p )
{
    ulonglong2 v;
    asm volatile( "ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"( v.x ), "=l"( v.y ) : "l"( p ) : "memory" );
    return v;
}

// The sums over all blocks of their N double-float words under `tag`, in every thread of the block;
// false when the wait ran out. The block's first warp polls (lane l blocks l, l + 32, ..., all at
// once) and adds up in a fixed order. ACQUIRE: what the blocks stored before they published is
// visible afterwards.
template <int N, bool ACQUIRE>
__device__ __forceinline__ bool meet( const ulonglong2* words, const PcgResidentArgs& a, uint32_t tag, DF* sum, float4* out )
{
    constexpr int kPer = 5;  // blocks per lane: up to 160
    if( threadIdx.x < 32 )
    {
        const int lane = threadIdx.x;
        ulonglong2 w[kPer][N];
        bool ok = false;
        for( unsigned n = 0;; ++n )  // (the loop's exit is a vote: uniform control flow)
        {
            ok = true;
#pragma unroll
            for( int q = 0; q < kPer; ++q )
            {
                const unsigned b = lane + 32 * q;
#pragma unroll
                for( int v = 0; v < N; ++v )
                    w[q][v] = b < a.expect ? load_words( words + (size_t)b * N + v ) : tagged( DF{ 0.f, 0.f }, tag );
            }
#pragma unroll
            for( int q = 0; q < kPer; ++q )
#pragma unroll
                for( int v = 0; v < N; ++v ) ok = ok && (uint32_t)( w[q][v].x >> 32 ) == tag && (uint32_t)( w[q][v].y >> 32 ) == tag;
            ok = __all_sync( 0xffffffffu, ok );
            if( ok || n >= a.limit ) break;
            if( ( n & 255u ) == 255u && __any_sync( 0xffffffffu, *(volatile uint32_t*)a.red.err != 0u ) ) break;
        }
        // one fence after the relaxed polls (acquiring loads would wait for one another), by every lane:
        // each has polled other blocks' words, and a fence orders what its own thread has read
        if( ACQUIRE ) asm volatile( "fence.acq_rel.gpu;" ::: "memory" );
        if( !ok && lane == 0 ) atomicOr( a.red.err, (uint32_t)BORA_REDUCE_ERR_BARRIER );
        DF t[2] = { { 0.f, 0.f }, { 0.f, 0.f } };
#pragma unroll
        for( int v = 0; v < N; ++v )
        {
#pragma unroll
            for( int q = 0; q < kPer; ++q )
                t[v] = df_add( t[v], DF{ __uint_as_float( (uint32_t)w[q][v].x ), __uint_as_float( (uint32_t)w[q][v].y ) } );
            t[v] = df_warp_sum_df( t[v] );
        }
        // a sum of squares is never negative: r.r = -1 (the second value) says that the wait ran out
        if( lane == 0 ) *out = ok ? make_float4( t[0].hi, t[0].lo, t[1].hi, t[1].lo ) : make_float4( 0.f, 0.f, -1.f, 0.f );
    }
    __syncthreads();
    const float4 o = *out;
    sum[0] = DF{ o.x, o.y };
    if( N > 1 ) sum[1] = DF{ o.z, o.w };
    return o.z != -1.f;
}

// The block's sums of N values published under `tag`. FENCE: everything its threads have stored is
// visible to a warp that acquires the words.
template <int W, int N, bool FENCE>
__device__ __forceinline__ void publish( ulonglong2* words, uint32_t tag, const DF* v, float2* w )
{
    DF t[N];
#pragma unroll
    for( int q = 0; q < N; ++q ) t[q] = df_warp_sum_df( v[q] );
    const int wid = threadIdx.x >> 5;
    if( ( threadIdx.x & 31 ) == 0 )
#pragma unroll
        for( int q = 0; q < N; ++q ) w[q * W + wid] = make_float2( t[q].hi, t[q].lo );
    __syncthreads();
    if( threadIdx.x == 0 )
    {
#pragma unroll
        for( int q = 0; q < N; ++q )
        {
            t[q] = DF{ w[q * W].x, w[q * W].y };
            for( int o = 1; o < W; ++o ) t[q] = df_add( t[q], DF{ w[q * W + o].x, w[q * W + o].y } );
        }
        if( FENCE ) asm volatile( "fence.acq_rel.gpu;" ::: "memory" );
#pragma unroll
        for( int q = 0; q < N; ++q ) store_words( words + (size_t)blockIdx.x * N + q, tagged( t[q], tag ) );
    }
    __syncwarp();  // lanes that went ahead to poll would hold up the one that publishes
}

template <int W>
__global__ void __launch_bounds__( 32 * W, 1 ) k_pcg_resident( const __grid_constant__ PcgResidentArgs a )
{
    __shared__ float2 s_sum[3][W];  // the warps' r.z and r.r; d.q
    __shared__ float4 s_met[2];     // the met sums
    constexpr unsigned kAll = 0xffffffffu;
    const int lane = threadIdx.x & 31, j = lane & 7, kq = lane >> 3;
    const int cA = 8 * ( j + 16 * kq );  // row A = (j, 2 kq); row B = (j, 2 kq + 1) 64 cells on
    const int t = blockIdx.x * W + ( threadIdx.x >> 5 );
    const bool mine = t < a.ft.n;
    float* const dg = a.dsel ? a.sv.d[1] : a.sv.d[0];
    int4 n0 = make_int4( -1, -1, -1, -1 ), n1 = n0;
    float rA[8], rB[8], dA[8], dB[8], eA[8], eB[8], mA[8], mB[8], zA[8], zB[8];
    uint4 wA = make_uint4( 0u, 0u, 0u, 0u ), wB = wA;
#pragma unroll
    for( int i = 0; i < 8; ++i ) rA[i] = rB[i] = dA[i] = dB[i] = eA[i] = eB[i] = mA[i] = mB[i] = 0.f;
    size_t g = 0;
    if( mine )
    {
        n0 = a.ft.tab[2 * t];
        n1 = a.ft.tab[2 * t + 1];
        g = (size_t)n1.z * 512 + cA;
        bora_ld8( a.sv.r + g, rA ); bora_ld8( a.sv.r + g + 64, rB );
        bora_ld8( a.sv.minv + g, mA ); bora_ld8( a.sv.minv + g + 64, mB );
        bora_ld8( dg + g, dA ); bora_ld8( dg + g + 64, dB );
        wA = *reinterpret_cast<const uint4*>( a.code + g );
        wB = *reinterpret_cast<const uint4*>( a.code + g + 64 );
    }
    // the neighbour tiles' cells that the lane's rows need: the x ends of both rows, the y face rows
    // of lanes j = 0 / 7, the z face row of row A at k = 0 and of row B at k = 7
    const int yt = j == 0 ? n0.z : ( j == 7 ? n0.w : -1 ), yc = cA + ( j == 0 ? 56 : -56 );
    const int zt = kq == 0 ? n1.x : ( kq == 3 ? n1.y : -1 ), zc = 8 * j + ( kq == 0 ? 448 : 0 );
    float hx[4], hyA[8], hyB[8], hz[8];  // their d
    auto halo = [&]( const float* v, float* x, float* yA, float* yB, float* z ) {
        auto one = [&]( int tl, int c ) { return tl < 0 ? 0.f : __ldcg( v + (size_t)tl * 512 + c ); };
        auto row = [&]( int tl, int c, float* o ) {
            const float4* p = reinterpret_cast<const float4*>( v + (size_t)( tl < 0 ? 0 : tl ) * 512 + ( tl < 0 ? 0 : c ) );
            const float4 zero = make_float4( 0.f, 0.f, 0.f, 0.f );
            const float4 l = tl < 0 ? zero : __ldcg( p ), h = tl < 0 ? zero : __ldcg( p + 1 );
            o[0] = l.x; o[1] = l.y; o[2] = l.z; o[3] = l.w; o[4] = h.x; o[5] = h.y; o[6] = h.z; o[7] = h.w;
        };
        x[0] = one( n0.x, cA + 7 ); x[1] = one( n0.y, cA ); x[2] = one( n0.x, cA + 71 ); x[3] = one( n0.y, cA + 64 );
        row( yt, yc, yA );
        row( yt, yc + 64, yB );
        row( zt, zc, z );
    };
    halo( dg, hx, hyA, hyB, hz );
    // z = M^-1 r, stored for the neighbours, and the sums r.z and r.r
    auto precondition = [&]( uint32_t tag ) {
        DF v[2] = { { 0.f, 0.f }, { 0.f, 0.f } };
#pragma unroll
        for( int h = 0; h < 8; h += 4 )
        {
            const float4 x = make_float4( rA[h], rA[h + 1], rA[h + 2], rA[h + 3] ), y = make_float4( rB[h], rB[h + 1], rB[h + 2], rB[h + 3] );
            v[1] = df_add_f( df_add_f( v[1], dot4( x, x ) ), dot4( y, y ) );
        }
#pragma unroll
        for( int i = 0; i < 8; ++i ) { zA[i] = rA[i]; zB[i] = rB[i]; }
        mic_sweeps<true>( zA, zB, mA, mB, v[0] );
        if( mine )
        {
            bora_st8( a.sv.z + g, zA );
            bora_st8( a.sv.z + g + 64, zB );
        }
        publish<W, 2, true>( a.words_rz, tag, v, &s_sum[0][0] );
    };
    uint32_t tag = a.tag;
    DF rz_prev{ 0.f, 0.f }, sum[2];
    bool cont = a.slot_rz_prev >= 0;  // the recurrence continues from d
    int last = a.max_inner, due = a.check;  // the pass's last iteration; the next one to be tested
    if( cont ) rz_prev = DF{ a.red.ringf[a.slot_rz_prev].x, a.red.ringf[a.slot_rz_prev].y };
#pragma unroll 1
    for( int it = 0;; ++it, ++tag )
    {
        precondition( tag );
        if( !meet<2, true>( a.words_rz, a, tag, sum, &s_met[0] ) ) return;
        const DF rz = sum[0], rr = sum[1];
        if( it == due )
        {
            due += a.check;
            if( __any_sync( kAll, !( rr.hi > a.above ) ) )
            {
                const double rrd = (double)rr.hi + (double)rr.lo;
                if( __any_sync( kAll, !( rrd > 0.0 ) || rrd <= a.target2 ) ) last = min( last, it + a.beyond );
            }
        }
        if( it >= last )
        {
            // the pass is done: it iterations
            if( mine )
            {
                bora_st8( dg + g, dA ); bora_st8( dg + g + 64, dB );
                bora_st8( a.sv.e + g, eA ); bora_st8( a.sv.e + g + 64, eB );
            }
            if( blockIdx.x == 0 && threadIdx.x == 0 )
            {
                ring_store( a.red, a.slot_a_rz, rz_prev, false );
                a.red.part_rr[0] = make_float2( rr.hi, rr.lo );  // finished by the refinement
                *(volatile uint32_t*)a.iters = (uint32_t)it;
            }
            return;
        }
        const float beta = cont ? df_ratio( make_float2( rz.hi, rz.lo ), make_float2( rz_prev.hi, rz_prev.lo ) ) : 0.f;
        float q[8], tA[8], qA[8];
        {
            float x[4], yA[8], yB[8], z[8];
            halo( a.sv.z, x, yA, yB, z );
#pragma unroll
            for( int i = 0; i < 8; ++i )
            {
                dA[i] = fmaf( beta, dA[i], zA[i] );
                dB[i] = fmaf( beta, dB[i], zB[i] );
                if( i < 4 ) hx[i] = fmaf( beta, hx[i], x[i] );
                hyA[i] = fmaf( beta, hyA[i], yA[i] );
                hyB[i] = fmaf( beta, hyB[i], yB[i] );
                hz[i] = fmaf( beta, hz[i], z[i] );
            }
        }
        auto stencil = [&]( const uint4& w, const float* d, const float* hy, const float* zm, const float* zp, float xm, float xp, float* o ) {
            const uint32_t cw[4] = { w.x, w.y, w.z, w.w };
#pragma unroll
            for( int i = 0; i < 8; ++i )
            {
                float ym = __shfl_up_sync( kAll, d[i], 1 ), yp = __shfl_down_sync( kAll, d[i], 1 );
                if( j == 0 ) ym = hy[i];
                if( j == 7 ) yp = hy[i];
                const uint32_t c = i & 1 ? cw[i >> 1] >> 16 : cw[i >> 1] & 0xffffu;
                o[i] = 0.f;
                if( c & BORA_CODE_FLUID )
                {
                    float acc = 0.f;
                    acc += i > 0 ? d[i > 0 ? i - 1 : 0] : xm; acc += i < 7 ? d[i < 7 ? i + 1 : 7] : xp;
                    acc += ym; acc += yp; acc += zm[i]; acc += zp[i];
                    o[i] = fmaf( (float)code_diag( (uint16_t)c ), d[i], -acc );
                }
            }
        };
        {
            float zm[8], zp[8];
#pragma unroll
            for( int i = 0; i < 8; ++i )
            {
                zm[i] = __shfl_up_sync( kAll, dB[i], 8 );
                zp[i] = __shfl_down_sync( kAll, dA[i], 8 );
                if( kq == 0 ) zm[i] = hz[i];
                if( kq == 3 ) zp[i] = hz[i];
            }
            stencil( wA, dA, hyA, zm, dB, hx[0], hx[1], qA );
            stencil( wB, dB, hyB, dA, zp, hx[2], hx[3], q );
        }
        DF pdq{ 0.f, 0.f };
#pragma unroll
        for( int i = 0; i < 8; ++i )
        {
            tA[i] = dA[i] * qA[i];
            pdq = df_add_f( pdq, fmaf( dB[i], q[i], tA[i] ) );
        }
        publish<W, 1, false>( a.words_dq, ++tag, &pdq, &s_sum[2][0] );
        DF dq;
        if( !meet<1, false>( a.words_dq, a, tag, &dq, &s_met[1] ) ) return;
        const float alpha = df_ratio( make_float2( rz.hi, rz.lo ), make_float2( dq.hi, dq.lo ) );
#pragma unroll
        for( int i = 0; i < 8; ++i )
        {
            eA[i] = fmaf( alpha, dA[i], eA[i] ); eB[i] = fmaf( alpha, dB[i], eB[i] );
            rA[i] = fmaf( -alpha, qA[i], rA[i] ); rB[i] = fmaf( -alpha, q[i], rB[i] );
        }
        rz_prev = rz;
        cont = true;
    }
}

// ---------------------------------------------------------------------------------
// float4 v of the solver's tiles -> its place in the cell vectors
__device__ __forceinline__ size_t solve_quad( const int4* tab, size_t v ) { return (size_t)solve_slot( tab, (int)( v >> 7 ) ) * 128 + ( v & 127 ); }

__device__ __forceinline__ void solve_init_body( const BoraSolveTilesDev& ft, const float* __restrict__ b, const BoraSolverDev& sv,
                                                 const BoraReduceDev& red, int slot_norm2, int slot_max, unsigned bid,
                                                 unsigned G )
{
    DF n2{ 0.f, 0.f };
    float mx = 0.f;
    const size_t n4 = (size_t)*ft.count * 128;
    for( size_t v = bid * (size_t)blockDim.x + threadIdx.x; v < n4; v += (size_t)G * blockDim.x )
    {
        const size_t i = solve_quad( ft.tab, v );
        const float4 bv = reinterpret_cast<const float4*>( b )[i], zero = make_float4( 0.f, 0.f, 0.f, 0.f );
        reinterpret_cast<float4*>( sv.r )[i] = bv;
        reinterpret_cast<float4*>( sv.x )[2 * i] = zero;
        reinterpret_cast<float4*>( sv.x )[2 * i + 1] = zero;
        reinterpret_cast<float4*>( sv.e )[i] = zero;
        reinterpret_cast<float4*>( sv.d[0] )[i] = zero;
        reinterpret_cast<float4*>( sv.q )[i] = zero;
        n2 = df_add( n2, df_prod( bv.x, bv.x ) );
        n2 = df_add( n2, df_prod( bv.y, bv.y ) );
        n2 = df_add( n2, df_prod( bv.z, bv.z ) );
        n2 = df_add( n2, df_prod( bv.w, bv.w ) );
        mx = fmaxf( fmaxf( mx, fmaxf( fabsf( bv.x ), fabsf( bv.y ) ) ), fmaxf( fabsf( bv.z ), fabsf( bv.w ) ) );
    }
    reduce2_publish_dfmax( n2, mx, red, slot_norm2, slot_max, bid, G );
}

// The warm start of a solve: x = the last step's pressure on fluid cells whose tile was active
// then (slot_prev: the previous tile table, virtual tile -> slot), 0 elsewhere.
__global__ void k_solve_warm( size_t ncells, const uint16_t* __restrict__ code, const int32_t* __restrict__ tile_of,
                              const int32_t* __restrict__ slot_prev, const float* __restrict__ pres, float2* __restrict__ x )
{
    for( size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < ncells; i += (size_t)gridDim.x * blockDim.x )
    {
        float v = 0.f;
        if( code[i] & BORA_CODE_FLUID )
        {
            const int os = slot_prev[tile_of[i >> 9]];
            if( os >= 0 ) v = pres[(size_t)os * BORA_TILE_CELLS + ( i & ( BORA_TILE_CELLS - 1 ) )];
        }
        x[i] = make_float2( v, 0.f );
    }
}

__global__ void k_solve_init( BoraSolveTilesDev ft, const float* __restrict__ b, BoraSolverDev sv, BoraReduceDev red,
                              int slot_norm2, int slot_max )
{
    solve_init_body( ft, b, sv, red, slot_norm2, slot_max, blockIdx.x, gridDim.x );
}

__global__ void k_solve_init_batch( const __grid_constant__ BoraBatchLaunch L )
{
    unsigned bid;
    const int k = bora_batch_member( L, blockIdx.x, &bid );
    const BoraMemberSolve& m = L.ms[k];
    const BoraMemberSlots& q = L.sl[k];
    solve_init_body( m.ft, m.b, m.sv, m.red, q.n2, q.mx, bid, (unsigned)m.grid[kGridCells] );
}

// x += e (+ the last update's pending alpha d), then clear e and q; the direction d is kept
// (the next refinement pass continues the recurrence from it).
__device__ __forceinline__ void refine_accumulate_body( const BoraSolveTilesDev& ft, const uint16_t* __restrict__ code,
                                                        const BoraSolverDev& sv, int dsel, const BoraReduceDev& red,
                                                        int nparts, int slot_rr, int slot_a_rz, int slot_a_dq, unsigned bid,
                                                        unsigned G )
{
    __shared__ float2 s_rr[8];  // 256 threads
    if( bid == G - 1 )          // the last update's r.r, for the host
    {
        const DF rr = part_collect( red.part_rr, nparts, s_rr );
        if( threadIdx.x == 0 ) ring_store( red, slot_rr, rr, true );
    }
    const bool pending = slot_a_rz >= 0;
    const float alpha = pending ? df_ratio( red.ringf[slot_a_rz], red.ringf[slot_a_dq] ) : 0.f;
    const float4* __restrict__ d = reinterpret_cast<const float4*>( dsel ? sv.d[1] : sv.d[0] );
    const size_t n4 = (size_t)ft.n * 128;
    for( size_t v = bid * (size_t)blockDim.x + threadIdx.x; v < n4; v += (size_t)G * blockDim.x )
    {
        const size_t i = solve_quad( ft.tab, v );
        const uint2 cw = reinterpret_cast<const uint2*>( code )[i];
        float4 e = reinterpret_cast<const float4*>( sv.e )[i];
        if( pending )
        {
            const float4 dv = d[i];
            e.x = fmaf( alpha, dv.x, e.x ); e.y = fmaf( alpha, dv.y, e.y );
            e.z = fmaf( alpha, dv.z, e.z ); e.w = fmaf( alpha, dv.w, e.w );
        }
        float4 x0 = reinterpret_cast<const float4*>( sv.x )[2 * i], x1 = reinterpret_cast<const float4*>( sv.x )[2 * i + 1];
        auto add = [&]( uint32_t c, float& hi, float& lo, float ev ) {
            if( !( c & BORA_CODE_FLUID ) ) return;
            const DF y = df_add_f( DF{ hi, lo }, ev );
            hi = y.hi;
            lo = y.lo;
        };
        add( cw.x, x0.x, x0.y, e.x );
        add( cw.x >> 16, x0.z, x0.w, e.y );
        add( cw.y, x1.x, x1.y, e.z );
        add( cw.y >> 16, x1.z, x1.w, e.w );
        reinterpret_cast<float4*>( sv.x )[2 * i] = x0;
        reinterpret_cast<float4*>( sv.x )[2 * i + 1] = x1;
        const float4 zero = make_float4( 0.f, 0.f, 0.f, 0.f );
        reinterpret_cast<float4*>( sv.e )[i] = zero;
        reinterpret_cast<float4*>( sv.q )[i] = zero;
    }
}

__global__ void k_refine_accumulate( BoraSolveTilesDev ft, const uint16_t* __restrict__ code, BoraSolverDev sv, int dsel,
                                     BoraReduceDev red, int nparts, int slot_rr, int slot_a_rz, int slot_a_dq )
{
    refine_accumulate_body( ft, code, sv, dsel, red, nparts, slot_rr, slot_a_rz, slot_a_dq, blockIdx.x, gridDim.x );
}

__global__ void k_refine_accumulate_batch( const __grid_constant__ BoraBatchLaunch L )
{
    unsigned bid;
    const int k = bora_batch_member( L, blockIdx.x, &bid );
    const BoraMemberSolve& m = L.ms[k];
    const BoraMemberSlots& q = L.sl[k];
    refine_accumulate_body( m.ft, m.code, m.sv, q.dsel, m.red, m.grid[kGridPass0R], q.rr_new, q.a_rz,
                            q.a_dq, bid, (unsigned)m.grid[kGridCells] );
}

// r = b - A x in double-float arithmetic (A from the stencil code, x the double-float iterate); r
// stored in FP32, ||r||^2 and max|r| reduced. One warp per half tile and a lane per x-row, as the
// direction kernel. GB300's FP64 pipe is narrow: in FP64 this kernel and the accumulation were
// bound by it. (A cell per thread with its neighbours' indices formed one by one: 54 us at 256^3,
// 35 now.)
constexpr int kResWarps = 8;

__device__ __forceinline__ void refine_residual_body( const BoraSolveTilesDev& ft, const float* __restrict__ b,
                                                      const uint16_t* __restrict__ code, const BoraSolverDev& sv, const BoraReduceDev& red, int slot_norm2,
                                                      int slot_max, unsigned bid, unsigned G )
{
    DF n2{ 0.f, 0.f };
    float mx = 0.f;
    const int lane = threadIdx.x & 31, j = lane & 7, kk = lane >> 3;
    const int nh = 2 * ft.n, stride = (int)G * kResWarps;
    constexpr unsigned kAll = 0xffffffffu;
    const float* __restrict__ x = reinterpret_cast<const float*>( sv.x );
    auto load = [&]( int t, int c, float* v ) {  // 8 double-float values
#pragma unroll
        for( int i = 0; i < 16; ++i ) v[i] = 0.f;
        if( t < 0 ) return;
        bora_ld8( x + 2 * ( (size_t)t * 512 + c ), v );
        bora_ld8( x + 2 * ( (size_t)t * 512 + c ) + 8, v + 8 );
    };
    // (a bound of the block's; a warp past the last half tile has no neighbours and stores nothing)
#pragma unroll 1
    for( int base = (int)bid * kResWarps; base < nh; base += stride )
    {
        const int h = base + (int)( threadIdx.x >> 5 );
        const bool mine = h < nh;
        const int t = mine ? h >> 1 : 0, hi = h & 1;
        int4 n0 = __ldg( ft.tab + 2 * (size_t)t ), n1 = __ldg( ft.tab + 2 * (size_t)t + 1 );
        const int s = n1.z;
        if( !mine ) n0 = n1 = make_int4( -1, -1, -1, -1 );
        const int cA = hi * 256 + 8 * lane;
        const size_t g = (size_t)s * 512 + cA;
        const int yt = j == 0 ? n0.z : ( j == 7 ? n0.w : -1 ), yc = cA + ( j == 0 ? 56 : -56 );
        const int sz = hi ? n1.y : n1.x, own = mine ? s : -1;
        const int zt = kk == 0 ? ( hi ? own : sz ) : ( kk == 3 ? ( hi ? sz : own ) : -1 );
        const int zc = 8 * j + ( kk == 0 ? ( hi ? 192 : 448 ) : ( hi ? 0 : 256 ) );
        uint4 cw = make_uint4( 0u, 0u, 0u, 0u );
        if( mine ) cw = *reinterpret_cast<const uint4*>( code + g );
        float v[16], yh[16], zh[16], bv[8] = {};
        load( own, cA, v );
        load( yt, yc, yh );
        load( zt, zc, zh );
        const float2 zero = make_float2( 0.f, 0.f );
        const float2 xm = n0.x < 0 ? zero : sv.x[(size_t)n0.x * 512 + cA + 7], xp = n0.y < 0 ? zero : sv.x[(size_t)n0.y * 512 + cA];
        if( mine ) bora_ld8( b + g, bv );
        const uint32_t w[4] = { cw.x, cw.y, cw.z, cw.w };
        float r[8];
        uint32_t seen = 0;
#pragma unroll
        for( int i = 0; i < 8; ++i )
        {
            const uint32_t c = i & 1 ? w[i >> 1] >> 16 : w[i >> 1] & 0xffffu;
            const float vh = v[2 * i], vl = v[2 * i + 1];
            float ymh = __shfl_up_sync( kAll, vh, 1 ), yml = __shfl_up_sync( kAll, vl, 1 );
            float yph = __shfl_down_sync( kAll, vh, 1 ), ypl = __shfl_down_sync( kAll, vl, 1 );
            float zmh = __shfl_up_sync( kAll, vh, 8 ), zml = __shfl_up_sync( kAll, vl, 8 );
            float zph = __shfl_down_sync( kAll, vh, 8 ), zpl = __shfl_down_sync( kAll, vl, 8 );
            if( j == 0 ) { ymh = yh[2 * i]; yml = yh[2 * i + 1]; }
            if( j == 7 ) { yph = yh[2 * i]; ypl = yh[2 * i + 1]; }
            if( kk == 0 ) { zmh = zh[2 * i]; zml = zh[2 * i + 1]; }
            if( kk == 3 ) { zph = zh[2 * i]; zpl = zh[2 * i + 1]; }
            // a neighbour that the code does not name counts as 0, which changes no sum
            DF acc{ 0.f, 0.f };
            auto add = [&]( int q, float nh_, float nl_ ) {
                const bool on = ( c >> q ) & 1u;
                acc = df_add( acc, DF{ on ? nh_ : 0.f, on ? nl_ : 0.f } );
            };
            add( 0, i ? v[i ? 2 * i - 2 : 0] : xm.x, i ? v[i ? 2 * i - 1 : 0] : xm.y );
            add( 1, i < 7 ? v[i < 7 ? 2 * i + 2 : 0] : xp.x, i < 7 ? v[i < 7 ? 2 * i + 3 : 0] : xp.y );
            add( 2, ymh, yml );
            add( 3, yph, ypl );
            add( 4, zmh, zml );
            add( 5, zph, zpl );
            const float dg = (float)code_diag( (uint16_t)c );
            const DF ax = df_add_f( df_prod( vh, dg ), vl * dg );  // diag * x (diag <= 12)
            const DF y = df_add( ax, DF{ -acc.hi, -acc.lo } );
            const DF rv = df_add_f( DF{ -y.hi, -y.lo }, bv[i] );
            const bool fluid = c & BORA_CODE_FLUID;
            r[i] = fluid ? rv.hi + rv.lo : 0.f;
            n2 = df_add( n2, df_prod( r[i], r[i] ) );
            mx = fmaxf( mx, fabsf( r[i] ) );
            if( fluid ) seen |= c & ( 0x3cu | ( i == 0 ? 1u : 0u ) | ( i == 7 ? 2u : 0u ) );
        }
        if( !mine ) continue;
        bora_st8( sv.r + g, r );
        // a code that names a fluid neighbour in an inactive tile is inconsistent (in an active tile
        // without fluid, where only a caller's codes name one, the neighbour counts as 0)
        auto bad = [&]( uint32_t bit, bool missing, int dir ) { return ( seen & bit ) && missing && ft.nbr[(size_t)s * 27 + dir] < 0; };
        if( bad( 1u, n0.x < 0, bora_dir( -1, 0, 0 ) ) || bad( 2u, n0.y < 0, bora_dir( 1, 0, 0 ) ) ||
            bad( 4u, j == 0 && yt < 0, bora_dir( 0, -1, 0 ) ) || bad( 8u, j == 7 && yt < 0, bora_dir( 0, 1, 0 ) ) ||
            bad( 16u, kk == 0 && zt < 0, bora_dir( 0, 0, -1 ) ) || bad( 32u, kk == 3 && zt < 0, bora_dir( 0, 0, 1 ) ) )
            atomicOr( red.err, 2u );
    }
    reduce2_publish_dfmax( n2, mx, red, slot_norm2, slot_max, bid, G );
}

__global__ void __launch_bounds__( 32 * kResWarps, 3 ) k_refine_residual( BoraSolveTilesDev ft, const float* __restrict__ b,
                                                            const uint16_t* __restrict__ code, BoraSolverDev sv,
                                                            BoraReduceDev red, int slot_norm2, int slot_max )
{
    refine_residual_body( ft, b, code, sv, red, slot_norm2, slot_max, blockIdx.x, gridDim.x );
}

__global__ void __launch_bounds__( 32 * kResWarps, 3 ) k_refine_residual_batch( const __grid_constant__ BoraBatchLaunch L )
{
    unsigned bid;
    const int k = bora_batch_member( L, blockIdx.x, &bid );
    const BoraMemberSolve& m = L.ms[k];
    const BoraMemberSlots& q = L.sl[k];
    refine_residual_body( m.ft, m.b, m.code, m.sv, m.red, q.n2, q.mx, bid,
                          (unsigned)m.grid[kGridResidual] );
}

__global__ void k_write_pressure( size_t ncells, const uint16_t* __restrict__ code, const float2* __restrict__ x,
                                  float* __restrict__ pres )
{
    for( size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < ncells; i += (size_t)gridDim.x * blockDim.x )
        pres[i] = ( code[i] & BORA_CODE_FLUID ) ? x[i].x + x[i].y : 0.f;
}

__global__ void k_write_pressure_batch( const __grid_constant__ BoraBatchLaunch L )
{
    unsigned bid;
    const BoraMemberSolve& m = L.ms[bora_batch_member( L, blockIdx.x, &bid )];
    const unsigned G = (unsigned)m.grid[kGridCells];
    const size_t ncells = (size_t)m.ntiles * 512;
    for( size_t i = bid * (size_t)blockDim.x + threadIdx.x; i < ncells; i += (size_t)G * blockDim.x )
        m.pres[i] = ( m.code[i] & BORA_CODE_FLUID ) ? m.sv.x[i].x + m.sv.x[i].y : 0.f;
}

// ---------------------------------------------------------------------------------
// Velocity update (FluidProjection.cu:293-378), in two passes over the half tiles: air cells next
// to fluid take the mean of their fluid neighbours' pressure, in place (the pass reads fluid
// cells' pressures only, and those it leaves alone); then fluid cells subtract the
// central-difference pressure gradient with the reference's ghost rules, other cells keep the
// P2G velocity. (One pass from a 12^3 staged region was bound by index arithmetic: 98 us at
// 256^3, 48 now.)

// sum of the fluid neighbours' pressures in the order -x +x -y +y -z +z over their number
struct AirMean
{
    float press = 0.f;
    int count = 0;
    __device__ __forceinline__ void add( bool in_grid, int flag, float p )
    {
        if( in_grid && flag == BORA_FLUID ) { press += p; count++; }
    }
    __device__ __forceinline__ float value() const { return count > 0 ? press / (float)count : 0.f; }
};

__global__ void __launch_bounds__( 32 * kRowWarps ) k_air_pressure( BoraGridDev g, BoraTilesDev t, int ntiles, BoraCellsDev c )
{
    const HalfRow r = half_row<kRowWarps>( g, t, ntiles );
    RowFlags f;
    f.load( g, c.flag, r );
    constexpr uint32_t kAllFluid = 0x01010101u * BORA_FLUID;
    if( __all_sync( 0xffffffffu, !r.mine || ( f.w.x == kAllFluid && f.w.y == kAllFluid ) ) ) return;
    const int own = r.mine ? r.s : -1;
    float p[8], pym[8], pyp[8], pzm[8], pzp[8], h[8];
    row8( c.pres, own, r.c, p );
    row8( c.pres, r.yt, r.yc, h );
    beside( p, h, 1, r.j == 0, r.j == 7, pym, pyp );
    row8( c.pres, r.zt, r.zc, h );
    beside( p, h, 8, r.kk == 0, r.kk == 3, pzm, pzp );
    const float pxm = r.xm < 0 ? 0.f : c.pres[(size_t)r.xm * BORA_TILE_CELLS + r.c + 7];
    const float pxp = r.xp < 0 ? 0.f : c.pres[(size_t)r.xp * BORA_TILE_CELLS + r.c];
    const int EI = g.nx - 1, EJ = g.ny - 1, EK = g.nz - 1;
    float out[8];
#pragma unroll
    for( int q = 0; q < 8; ++q )
    {
        const int I = r.i0 + q, own_flag = flag_of( f.w, q );
        AirMean m;
        m.add( I > 0, q ? flag_of( f.w, q ? q - 1 : 0 ) : f.xm, q ? p[q ? q - 1 : 0] : pxm );
        m.add( I < EI, q < 7 ? flag_of( f.w, q < 7 ? q + 1 : 7 ) : f.xp, q < 7 ? p[q < 7 ? q + 1 : 7] : pxp );
        m.add( r.J > 0, flag_of( f.ym, q ), pym[q] );
        m.add( r.J < EJ, flag_of( f.yp, q ), pyp[q] );
        m.add( r.K > 0, flag_of( f.zm, q ), pzm[q] );
        m.add( r.K < EK, flag_of( f.zp, q ), pzp[q] );
        out[q] = own_flag == BORA_FLUID ? p[q] : ( own_flag == BORA_AIR && f.in_grid[q >> 2] ? m.value() : 0.f );
    }
    if( !r.mine ) return;
    // fluid cells are not stored: other warps read them
#pragma unroll
    for( int q = 0; q < 8; ++q )
        if( flag_of( f.w, q ) != BORA_FLUID ) c.pres[r.at() + q] = out[q];
}

// The air pressure of cell (i, j, k), which lies in the grid and in an inactive tile (only where
// the caller has set flags: the tiles around every particle are active), out of line.
__device__ __noinline__ float air_pressure_at( const BoraGridDev* g, const int32_t* slot_of, const uint8_t* flag,
                                               const float* pres, int i, int j, int k )
{
    AirMean m;
    for( int q = 0; q < 6; ++q )
    {
        const int n[3] = { i + ( q == 0 ? -1 : q == 1 ? 1 : 0 ), j + ( q == 2 ? -1 : q == 3 ? 1 : 0 ), k + ( q == 4 ? -1 : q == 5 ? 1 : 0 ) };
        if( n[0] < 0 || n[1] < 0 || n[2] < 0 || n[0] >= g->nx || n[1] >= g->ny || n[2] >= g->nz ) continue;
        const int s = slot_of[( (size_t)( n[2] >> 3 ) * g->ty + ( n[1] >> 3 ) ) * g->tx + ( n[0] >> 3 )];
        if( s < 0 ) continue;
        const size_t cell = (size_t)s * BORA_TILE_CELLS + bora_local( n[0], n[1], n[2] );
        m.add( true, flag[cell], pres[cell] );
    }
    return m.value();
}

__global__ void __launch_bounds__( 32 * kRowWarps ) k_vel_update( const __grid_constant__ BoraGridDev g, BoraTilesDev t, int ntiles,
                                                                  BoraCellsDev c )
{
    const HalfRow r = half_row<kRowWarps>( g, t, ntiles );
    RowFlags f;
    f.load( g, c.flag, r );
    const int own = r.mine ? r.s : -1;
    float p[8], pym[8], pyp[8], pzm[8], pzp[8], yh[8], zh[8], vx[8], vy[8], vz[8];
    row8( c.pres, own, r.c, p );
    row8( c.pres, r.yt, r.yc, yh );
    row8( c.pres, r.zt, r.zc, zh );
    float pxm = r.xm < 0 ? 0.f : c.pres[(size_t)r.xm * BORA_TILE_CELLS + r.c + 7];
    float pxp = r.xp < 0 ? 0.f : c.pres[(size_t)r.xp * BORA_TILE_CELLS + r.c];
    row8( c.vx, own, r.c, vx );
    row8( c.vy, own, r.c, vy );
    row8( c.vz, own, r.c, vz );
    const int EI = g.nx - 1, EJ = g.ny - 1, EK = g.nz - 1;
    // fluid cells next to an inactive tile
    if( r.mine )
    {
        auto outside = [&]( int i, int j, int k ) { return air_pressure_at( &g, t.slot_of, c.flag, c.pres, i, j, k ); };
        if( r.xm < 0 && r.i0 > 0 && flag_of( f.w, 0 ) == BORA_FLUID ) pxm = outside( r.i0 - 1, r.J, r.K );
        if( r.xp < 0 && r.i0 + 7 < EI && flag_of( f.w, 7 ) == BORA_FLUID ) pxp = outside( r.i0 + 8, r.J, r.K );
        const int dy = r.j == 0 ? -1 : 1, dz = r.kk == 0 ? -1 : 1;
        const bool y_out = ( r.j == 0 || r.j == 7 ) && r.yt < 0 && r.J + dy >= 0 && r.J + dy <= EJ;
        const bool z_out = ( r.kk == 0 || r.kk == 3 ) && r.zt < 0 && r.K + dz >= 0 && r.K + dz <= EK;
        if( y_out || z_out )
#pragma unroll
            for( int q = 0; q < 8; ++q )
            {
                if( flag_of( f.w, q ) != BORA_FLUID ) continue;
                if( y_out ) yh[q] = outside( r.i0 + q, r.J + dy, r.K );
                if( z_out ) zh[q] = outside( r.i0 + q, r.J, r.K + dz );
            }
    }
    beside( p, yh, 1, r.j == 0, r.j == 7, pym, pyp );
    beside( p, zh, 8, r.kk == 0, r.kk == 3, pzm, pzp );
    const int wall = (float)r.J + 0.5f <= g.voxel_wall + 1.f ? BORA_SOLID : BORA_AIR;
#pragma unroll
    for( int q = 0; q < 8; ++q )
    {
        const int own_flag = flag_of( f.w, q );
        const bool e_i0 = r.i0 + q == 0, e_i1 = r.i0 + q == EI, e_j0 = r.J == 0, e_j1 = r.J == EJ, e_k0 = r.K == 0, e_k1 = r.K == EK;
        auto grad = [&]( float lo, float hi, bool e0, bool e1, int t0, int t1 ) {
            t0 = e0 ? wall : t0;
            t1 = e1 ? wall : t1;
            const float n0 = e0 ? 2.f * p[q] - hi : lo, n1 = e1 ? 2.f * p[q] - lo : hi;
            const float a = t0 == BORA_SOLID ? 2.f * p[q] - n1 : t0 == BORA_AIR ? -n0 : n0;
            const float b = t1 == BORA_SOLID ? 2.f * p[q] - n0 : t1 == BORA_AIR ? -n1 : n1;
            return ( b - a ) * 0.5f;
        };
        const float dx = grad( q ? p[q ? q - 1 : 0] : pxm, q < 7 ? p[q < 7 ? q + 1 : 7] : pxp, e_i0, e_i1,
                               q ? flag_of( f.w, q ? q - 1 : 0 ) : f.xm, q < 7 ? flag_of( f.w, q < 7 ? q + 1 : 7 ) : f.xp );
        const float dy = grad( pym[q], pyp[q], e_j0, e_j1, flag_of( f.ym, q ), flag_of( f.yp, q ) );
        const float dz = grad( pzm[q], pzp[q], e_k0, e_k1, flag_of( f.zm, q ), flag_of( f.zp, q ) );
        const bool fluid = own_flag == BORA_FLUID, masked = own_flag == BORA_MASKED;
        vx[q] = masked ? 0.f : ( fluid ? vx[q] - dx : vx[q] );
        vy[q] = masked ? 0.f : ( fluid ? vy[q] - dy : vy[q] );
        vz[q] = masked ? 0.f : ( fluid ? vz[q] - dz : vz[q] );
    }
    if( !r.mine ) return;
    bora_st8( c.cx + r.at(), vx );
    bora_st8( c.cy + r.at(), vy );
    bora_st8( c.cz + r.at(), vz );
}

int grid_for( size_t n, int threads )
{
    const size_t b = ( n + threads - 1 ) / threads;
    return (int)( b < 152 * 8 ? ( b > 0 ? b : 1 ) : 152 * 8 );
}

}  // namespace

void bora_launch_rhs( const BoraGridDev& g, int ntiles, BoraTilesDev t, BoraCellsDev c, uint32_t* nfluid, uint8_t* tile_fluid,
                      cudaStream_t st )
{
    if( ntiles > 0 ) k_rhs<<<row_grid( ntiles, kRowWarps ), 32 * kRowWarps, 0, st>>>( g, t, ntiles, c, nfluid, tile_fluid );
}

void bora_launch_tile_fluid( int ntiles, const uint16_t* code, uint8_t* tile_fluid, cudaStream_t st )
{
    if( ntiles > 0 ) k_tile_fluid<<<grid_for( (size_t)ntiles * 32, 256 ), 256, 0, st>>>( ntiles, code, tile_fluid );
}

void bora_launch_flag_list( int n, const uint8_t* flags, int32_t* list, int stride, int offset, uint32_t* count,
                            uint32_t* host_count, cudaStream_t st )
{
    k_flag_list<<<1, 1024, 0, st>>>( n, flags, list, stride, offset, count, host_count );
}

void bora_launch_solve_tiles( int ntiles, BoraTilesDev t, const uint8_t* tile_fluid, int4* tab, uint32_t* count,
                              uint32_t* host_count, cudaStream_t st )
{
    bora_launch_flag_list( ntiles, tile_fluid, reinterpret_cast<int32_t*>( tab ), 8, 6, count, host_count, st );
    if( ntiles > 0 )
        k_solve_nbrs<<<grid_for( (size_t)ntiles * 8, 256 ), 256, 0, st>>>( count, t.nbr, tile_fluid, reinterpret_cast<int32_t*>( tab ) );
}

void bora_launch_vel_update( const BoraGridDev& g, int ntiles, BoraTilesDev t, BoraCellsDev c, cudaStream_t st )
{
    if( ntiles <= 0 ) return;
    k_air_pressure<<<row_grid( ntiles, kRowWarps ), 32 * kRowWarps, 0, st>>>( g, t, ntiles, c );
    k_vel_update<<<row_grid( ntiles, kRowWarps ), 32 * kRowWarps, 0, st>>>( g, t, ntiles, c );
}

void bora_launch_mic_factor( int ntiles, BoraSolveTilesDev t, const uint16_t* code, float* minv, cudaStream_t st )
{
    ensure_tables();
    if( ntiles <= 0 ) return;
    const int nb = std::min( ( ntiles + kTilesPerCta - 1 ) / kTilesPerCta, num_sms() * 8 );
    k_mic_factor<<<nb, 32 * kTilesPerCta, 0, st>>>( t, code, minv );
}

void bora_launch_solve_init( int ntiles, BoraSolveTilesDev t, const float* b, BoraSolverDev s, BoraReduceDev red,
                             int slot_norm2, int slot_max, cudaStream_t st )
{
    k_solve_init<<<grid_for( (size_t)ntiles * 128, 256 ), 256, 0, st>>>( t, b, s, red, slot_norm2, slot_max );
}

int bora_pcg_update_grid( int ntiles )
{
    static BoraPerDevice per_sm;
    const int bps = per_sm.get( [] {
        int v = 0;
        return cudaOccupancyMaxActiveBlocksPerMultiprocessor( &v, k_pcg_update, 32 * kUpdWarps, 0 ) == cudaSuccess && v > 0 ? v : 1;
    } );
    // as many rounds of one tile per warp as the resident warps need, and the grid sized so
    // that every warp gets that many tiles (no warp waits in the reduction for a straggler)
    const int cap = std::max( 1, std::min( bps * num_sms(), kBoraMaxReduceBlocks ) ) * kUpdWarps;
    const int rounds = std::max( 1, ( ntiles + cap - 1 ) / cap );  // one block even for no tiles: it publishes the sums
    return std::max( 1, ( ntiles + kUpdWarps * rounds - 1 ) / ( kUpdWarps * rounds ) );
}

void bora_launch_pcg_update( BoraSolveTilesDev t, BoraSolverDev s, BoraReduceDev red, int slot_rz_in, int slot_dq_in,
                             cudaStream_t st )
{
    bora_launch_pdl( k_pcg_update, bora_pcg_update_grid( t.n ), 32 * kUpdWarps, 0, st, t, s, red, bora_pcg_direction_grid( t.n ),
                     slot_rz_in, slot_dq_in );
}

// Grid of the direction kernel: every warp gets the same number of half tiles; at most
// kBoraMaxReduceBlocks CTAs (partial sums capacity).
int bora_pcg_direction_grid( int ntiles )
{
    if( ntiles <= 0 ) return 0;
    static BoraPerDevice per_sm;
    const int b = per_sm.get( [] {
        int v = 0;
        return cudaOccupancyMaxActiveBlocksPerMultiprocessor( &v, k_pcg_direction, 32 * kDirWarps, 0 ) == cudaSuccess && v > 0 ? v : 1;
    } );
    const int cap = std::max( 1, std::min( b * num_sms(), kBoraMaxReduceBlocks ) ) * kDirWarps;
    const int rounds = ( 2 * ntiles + cap - 1 ) / cap;
    return std::max( 1, ( 2 * ntiles + kDirWarps * rounds - 1 ) / ( kDirWarps * rounds ) );
}

namespace {
// equal rounds of the warps that are resident (three CTAs per SM at 80 registers)
int residual_grid( int nft )
{
    const int cap = 3 * num_sms() * kResWarps, rounds = std::max( 1, ( 2 * nft + cap - 1 ) / cap );
    return std::max( 1, ( 2 * nft + kResWarps * rounds - 1 ) / ( kResWarps * rounds ) );
}
}  // namespace

void bora_projection_grids( int nft, int* grid )
{
    grid[kGridDir] = bora_pcg_direction_grid( nft );
    grid[kGridCells] = grid_for( (size_t)nft * 128, 256 );
    grid[kGridResidual] = residual_grid( nft );
}

void bora_launch_solve_init_batch( const BoraBatchLaunch& L, int blocks, cudaStream_t st )
{
    if( blocks > 0 ) k_solve_init_batch<<<blocks, 256, 0, st>>>( L );
}

void bora_launch_pcg_direction_batch( const BoraBatchLaunch& L, int blocks, cudaStream_t st )
{
    if( blocks > 0 ) bora_launch_pdl( k_pcg_direction_batch, dim3( blocks ), dim3( 32 * kDirWarps ), 0, st, L );
}

void bora_launch_refine_accumulate_batch( const BoraBatchLaunch& L, int blocks, cudaStream_t st )
{
    if( blocks > 0 ) k_refine_accumulate_batch<<<blocks, 256, 0, st>>>( L );
}

void bora_launch_refine_residual_batch( const BoraBatchLaunch& L, int blocks, cudaStream_t st )
{
    if( blocks > 0 ) k_refine_residual_batch<<<blocks, 256, 0, st>>>( L );
}

void bora_launch_write_pressure_batch( const BoraBatchLaunch& L, int blocks, cudaStream_t st )
{
    if( blocks > 0 ) k_write_pressure_batch<<<blocks, 256, 0, st>>>( L );
}

int bora_pcg_persistent_grid()
{
    static BoraPerDevice per_sm;
    const int b = per_sm.get( [] {
        int v = 0;
        return cudaOccupancyMaxActiveBlocksPerMultiprocessor( &v, k_pcg_persistent, 32 * kUpdWarps, 0 ) == cudaSuccess ? v : 0;
    } );
    return std::min( b * num_sms(), kBoraMaxReduceBlocks );
}

int bora_launch_pcg_persistent( BoraSolveTilesDev t, const uint16_t* code, BoraSolverDev s, BoraReduceDev red,
                                int dsel, int slot_rz_prev, int max_inner, double target, int slot_a_rz, int slot_a_dq,
                                uint32_t* iters, unsigned* bar, double* part, bool never_release, cudaStream_t st )
{
    const int grid = bora_pcg_persistent_grid();
    if( grid <= 0 ) return -1;
    PcgPersistArgs a{};
    a.ft = t; a.code = code; a.sv = s; a.red = red;
    a.dsel = dsel; a.slot_rz_prev = slot_rz_prev; a.max_inner = max_inner; a.target = target;
    a.slot_a_rz = slot_a_rz; a.slot_a_dq = slot_a_dq; a.iters = iters;
    a.bar = bar; a.part = part;
    // a barrier that waits for one block more than there are never releases: every wait runs
    // out (fault injection for tests), after a short limit
    a.expect = (unsigned)grid + ( never_release ? 1u : 0u );
    a.limit = never_release ? ( 1u << 12 ) : ( 1u << 22 );
    if( cudaMemsetAsync( bar, 0, 2 * sizeof( unsigned ), st ) != cudaSuccess ) return -1;
    void* args[] = { &a };
    return cudaLaunchCooperativeKernel( (const void*)k_pcg_persistent, dim3( grid ), dim3( 32 * kUpdWarps ), args, 0, st ) ==
                   cudaSuccess
               ? 0
               : -1;
}

namespace {
// One warp per SM partition up to 256 tiles; above, two, as the blocks poll one another and the
// meetings grow with their number (464 tiles: 11.2 us per iteration in 116 blocks, 9.6 in 58).
constexpr int kResidentTiles4 = 256, kResidentTiles8 = 608;
constexpr int kResidentBlocks = std::max( ( kResidentTiles4 + 3 ) / 4, ( kResidentTiles8 + 7 ) / 8 );  // the largest grid (meet: 160)

// blocks of k_pcg_resident<W> that the device can run at once
template <int W>
int resident_blocks()
{
    static BoraPerDevice per_sm;
    const int b = per_sm.get( [] {
        int v = 0;
        return cudaOccupancyMaxActiveBlocksPerMultiprocessor( &v, k_pcg_resident<W>, 32 * W, 0 ) == cudaSuccess && v > 0 ? v : -1;
    } );
    return b > 0 ? b * num_sms() : 0;
}
}  // namespace

// Warps per block, 0: not for this form (too many tiles, or the device cannot run the grid at once). The
// step's GPU time against the per-phase form: 0.45 against 0.58 ms at 18 solver tiles, 1.10 against 1.28
// at 196, 1.43 against 1.60 at 356, 1.82 against 1.88 at 488, 2.05 against 2.11 at 632, level at 715 (2.28
// and 2.25) and 776 (2.51 and 2.54): the line lies where it stops to gain, at four tiles per SM.
int bora_pcg_resident_warps( int nft )
{
    if( nft <= 0 || nft > kResidentTiles8 ) return 0;
    if( nft <= kResidentTiles4 ) return resident_blocks<4>() >= ( nft + 3 ) / 4 ? 4 : 0;
    return resident_blocks<8>() >= ( nft + 7 ) / 8 ? 8 : 0;
}

size_t bora_pcg_resident_words_bytes() { return (size_t)3 * ( kResidentBlocks + 8 ) * sizeof( ulonglong2 ); }

int bora_launch_pcg_resident( BoraSolveTilesDev t, const uint16_t* code, BoraSolverDev s, BoraReduceDev red, int dsel,
                              int slot_rz_prev, int max_inner, int check, int beyond, double target, int slot_a_rz,
                              uint32_t* iters, void* words, uint32_t tag, bool never_release, cudaStream_t st )
{
    const int W = bora_pcg_resident_warps( t.n );
    if( W == 0 ) return -1;
    PcgResidentArgs a{};
    a.ft = t; a.code = code; a.sv = s; a.red = red; a.dsel = dsel; a.slot_rz_prev = slot_rz_prev; a.max_inner = max_inner;
    a.check = check;
    a.beyond = beyond;
    a.target2 = target * target;
    a.above = (float)( a.target2 * ( 1.0 + 1e-6 ) );
    a.slot_a_rz = slot_a_rz; a.iters = iters;
    a.words_rz = static_cast<ulonglong2*>( words );
    a.words_dq = a.words_rz + 2 * ( kResidentBlocks + 8 );
    a.tag = tag;
    const int grid = ( t.n + W - 1 ) / W;
    // a meeting that waits for one block more than there are never ends: every wait runs out (fault
    // injection for tests), after a short limit
    a.expect = (unsigned)grid + ( never_release ? 1u : 0u );
    a.limit = never_release ? ( 1u << 12 ) : ( 1u << 21 );
    void* args[] = { &a };
    const void* k = W == 4 ? (const void*)k_pcg_resident<4> : (const void*)k_pcg_resident<8>;
    return cudaLaunchCooperativeKernel( k, dim3( grid ), dim3( 32 * W ), args, 0, st ) == cudaSuccess ? 0 : -1;
}

void bora_launch_pcg_direction( BoraSolveTilesDev t, const uint16_t* code, BoraSolverDev s, int dsel_in, BoraReduceDev red, int nparts, int slot_rz_new, int slot_rr, int slot_rz_old,
                                int slot_a_rz, int slot_a_dq, bool host_rr, cudaStream_t st )
{
    if( t.n <= 0 ) return;
    bora_launch_pdl( k_pcg_direction, bora_pcg_direction_grid( t.n ), 32 * kDirWarps, 0, st, t, code, s, dsel_in, red, nparts, slot_rz_new, slot_rr, slot_rz_old, slot_a_rz, slot_a_dq, host_rr );
}

void bora_launch_solve_warm( int ntiles, const uint16_t* code, const int32_t* tile_of, const int32_t* slot_prev,
                             const float* pres, BoraSolverDev s, cudaStream_t st )
{
    const size_t nc = (size_t)ntiles * 512;
    if( nc ) k_solve_warm<<<grid_for( nc, 256 ), 256, 0, st>>>( nc, code, tile_of, slot_prev, pres, s.x );
}

void bora_launch_refine_accumulate( BoraSolveTilesDev t, const uint16_t* code, BoraSolverDev s, int dsel, BoraReduceDev red,
                                    int nparts, int slot_rr, int slot_a_rz, int slot_a_dq, cudaStream_t st )
{
    if( t.n > 0 )
        k_refine_accumulate<<<grid_for( (size_t)t.n * 128, 256 ), 256, 0, st>>>( t, code, s, dsel, red, nparts, slot_rr, slot_a_rz,
                                                                              slot_a_dq );
}

void bora_launch_refine_residual( BoraSolveTilesDev t, const float* b, const uint16_t* code, BoraSolverDev s, BoraReduceDev red,
                                  int slot_norm2, int slot_max, cudaStream_t st )
{
    k_refine_residual<<<residual_grid( t.n ), 32 * kResWarps, 0, st>>>( t, b, code, s, red, slot_norm2, slot_max );
}

void bora_launch_write_pressure( int ntiles, const uint16_t* code, const float2* x, float* pres, cudaStream_t st )
{
    const size_t nc = (size_t)ntiles * 512;
    if( nc ) k_write_pressure<<<grid_for( nc, 256 ), 256, 0, st>>>( nc, code, x, pres );
}
