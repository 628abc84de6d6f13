// Geometric multigrid V-cycle preconditioner for the pressure PCG, with FP16 storage
// and FP32 arithmetic (the mixed-precision form of the projection).
//
// The reference's pressure solve is unpreconditioned FP32 CG
// (base/source/LinearSystemSolver.cpp:12-50); its only preconditioner is a serial MIC(0)
// (base/source/BLAS.cu:211-331). This V-cycle replaces both for the mixed form.
//
// Hierarchy: level 0 is the fine grid of active 8^3 tiles; levels 1..3 keep the tile
// layout with 4^3, 2^3 and 1 cell per tile (neighbours across tiles through the tile
// neighbour table); levels >= 4 are small dense grids over the tile grid halved per
// level. A coarse cell is air (Dirichlet) if any child is air (inactive tiles count as
// air), else fluid if any child is fluid, else solid. Every level applies the reference's
// 7-point rule (diagonal 6 + #air - #solid/wall, -1 per fluid neighbour,
// FluidProjection.cu:234-244) to its own cell types; coarse operators are the
// rediscretisation with spacing 2^l, i.e. the same stencil divided by 4^l.
//
// All quantities are kept in "stencil units" (the level equation S z = r' with
// S = diag*z - sum of fluid neighbours): restriction averages the children's residuals
// and multiplies by 4, prolongation injects the coarse correction. Smoothing is two
// Jacobi sweeps before and after with Chebyshev weights (kOmegaA, kOmegaB below); the
// coarsest level (<= 512 cells) gets 16 damped Jacobi sweeps. Level residuals and corrections are stored as FP16: the fine residual
// is scaled by 1/||r||_2 on entry so every stored value is O(1). Residuals restricted to
// non-fluid coarse cells are never read (their z is zero), so the restriction does not
// look at the coarse types.
#include <algorithm>

#include <cuda_fp16.h>

#include "bora_internal.h"
#include "reduce.cuh"

namespace {

// Smoothing: the two Jacobi sweeps of each pre- and post-smoother take the weights of the
// degree-2 Chebyshev polynomial in D^-1 A over [0.35, 2] (roots 1.175 -+ 0.825 cos(pi/4)):
// the pre-smoother sweeps with kOmegaA then kOmegaB, the post-smoother with kOmegaB then
// kOmegaA. The two factors commute, so each level's post-smoother is the adjoint of its
// pre-smoother and the V-cycle stays symmetric. Against two sweeps of damped Jacobi
// (omega 0.9) this cut the PCG iterations of the dam-break scenes by a fifth at the same
// cost per V-cycle. The coarsest level keeps damped Jacobi with kOmega.
constexpr float kOmega = 0.9f;
constexpr float kOmegaA = 0.5687f;  // 1 / (1.175 + 0.825 cos(pi/4))
constexpr float kOmegaB = 1.6902f;  // 1 / (1.175 - 0.825 cos(pi/4))

__device__ inline int code_diag( uint16_t c ) { return ( c >> 8 ) & 15; }

// ---- set-up: cell types and stencil codes of coarse levels ---------------------------
//
// A coarse cell is air when one of its children is, else fluid when one is, else solid; beyond
// the domain it is masked. Children beyond the finer level's domain count as none (wall-like).
// Three launches: the tiled levels' types, the dense levels' types, all levels' codes (with two
// launches a level and a cell per thread the set-up was 8 to 14 launches. With the right-hand side
// and the solver's tile table: 83 -> 50 us at 96^3, 155 -> 94 at 256^3, 237 -> 136 in a 640 tank.)
// dense cells up to which one CTA forms a level's types (the 4096 of a 256^3 grid: 102 us in one CTA
// with the right-hand side, 94 over the grid)
constexpr size_t kDenseOneCta = 2048;

struct SetupLevels
{
    BoraLevelDev L[16];
    int n;
    const int32_t* nbr;
    const int32_t* slot_of;
    const int32_t* tile_of;
    int tx, ty, tz;
    float voxel_wall;
};

__device__ __forceinline__ int coarse_type( bool air, bool fluid ) { return air ? BORA_AIR : ( fluid ? BORA_FLUID : BORA_SOLID ); }

// Types of levels 1, 2, 3 (4^3, 2^3, 1 cells per tile), 16 lanes per tile: a lane owns the four
// level-1 cells of a row (y, z), lane = y + 4 z.
__global__ void __launch_bounds__( 256 ) k_mg_types_tiled( const __grid_constant__ SetupLevels d, int ntiles )
{
    const int s0 = (int)( ( blockIdx.x * (size_t)blockDim.x + threadIdx.x ) >> 4 ), s = min( s0, ntiles - 1 );
    const bool mine = s0 < ntiles;
    const int y = threadIdx.x & 3, z = ( threadIdx.x >> 2 ) & 3;
    const int vt = d.tile_of[s];
    const int ti = vt % d.tx, tj = ( vt / d.tx ) % d.ty, tk = vt / ( d.tx * d.ty );
    const BoraLevelDev& F = d.L[0];
    uint32_t air = 0, fluid = 0;  // bit x: a child of cell x is air / fluid
#pragma unroll
    for( int o = 0; o < 4; ++o )
    {
        const int b = 2 * y + ( o & 1 ), c = 2 * z + ( o >> 1 );
        if( tj * 8 + b >= F.ny || tk * 8 + c >= F.nz ) continue;
        const uint2 w = *reinterpret_cast<const uint2*>( F.type + (size_t)s * 512 + 8 * b + 64 * c );
#pragma unroll
        for( int a = 0; a < 8; ++a )
        {
            const int t = (int)( ( ( a < 4 ? w.x : w.y ) >> ( 8 * ( a & 3 ) ) ) & 255u );
            if( ti * 8 + a >= F.nx ) continue;
            if( t == BORA_AIR ) air |= 1u << ( a >> 1 );
            else if( t == BORA_FLUID ) fluid |= 1u << ( a >> 1 );
        }
    }
    int n = 4;  // the level's cells along the row and per tile edge
#pragma unroll
    for( int l = 1; l <= 3; ++l )
    {
        if( l >= d.n || d.L[l].kind != 0 ) return;
        const BoraLevelDev& C = d.L[l];
        const int step = 1 << ( l - 1 ), yy = y / step, zz = z / step;
        uint32_t types = 0, na = 0, nf = 0;
        for( int x = 0; x < n; ++x )
        {
            const bool real = ti * n + x < C.nx && tj * n + yy < C.ny && tk * n + zz < C.nz;
            const int t = real ? coarse_type( ( air >> x ) & 1u, ( fluid >> x ) & 1u ) : BORA_MASKED;
            types |= (uint32_t)t << ( 8 * x );
            if( t == BORA_AIR ) na |= 1u << ( x >> 1 );
            else if( t == BORA_FLUID ) nf |= 1u << ( x >> 1 );
        }
        if( mine && !( y & ( step - 1 ) ) && !( z & ( step - 1 ) ) )
        {
            uint8_t* out = C.type + (size_t)s * ( n * n * n ) + n * ( yy + n * zz );
            if( n == 4 ) *reinterpret_cast<uint32_t*>( out ) = types;
            else if( n == 2 ) *reinterpret_cast<uint16_t*>( out ) = (uint16_t)types;
            else *out = (uint8_t)types;
        }
        // the next level's children: the cells of the row and of the rows y, z + step
        air = na;
        fluid = nf;
        air |= __shfl_xor_sync( 0xffffffffu, air, step );
        fluid |= __shfl_xor_sync( 0xffffffffu, fluid, step );
        air |= __shfl_xor_sync( 0xffffffffu, air, 4 * step );
        fluid |= __shfl_xor_sync( 0xffffffffu, fluid, 4 * step );
        n >>= 1;
    }
}

// Type of cell `cell` of dense level l from the finer level (dense, or level 3: tiles).
__device__ __forceinline__ void dense_type( const SetupLevels& d, int l, long long cell )
{
    const BoraLevelDev &C = d.L[l], &F = d.L[l - 1];
    const int i = (int)( cell % C.dx ), j = (int)( ( cell / C.dx ) % C.dy ), k = (int)( cell / ( (long long)C.dx * C.dy ) );
    if( i >= C.nx || j >= C.ny || k >= C.nz ) { C.type[cell] = BORA_MASKED; return; }
    int t[8];
#pragma unroll
    for( int o = 0; o < 8; ++o )
    {
        const int a = 2 * i + ( o & 1 ), b = 2 * j + ( ( o >> 1 ) & 1 ), c = 2 * k + ( o >> 2 );
        t[o] = BORA_MASKED;
        if( a >= F.nx || b >= F.ny || c >= F.nz ) continue;
        if( F.kind == 1 ) t[o] = F.type[(long long)a + (long long)F.dx * ( b + (long long)F.dy * c )];
        else if( a < d.tx && b < d.ty && c < d.tz )
        {
            const int s = d.slot_of[( (size_t)c * d.ty + b ) * d.tx + a];
            t[o] = s < 0 ? BORA_AIR : F.type[s];
        }
    }
    bool air = false, fluid = false;
#pragma unroll
    for( int o = 0; o < 8; ++o )
    {
        air = air || t[o] == BORA_AIR;
        fluid = fluid || t[o] == BORA_FLUID;
    }
    C.type[cell] = (uint8_t)coarse_type( air, fluid );
}

// Types of dense levels [first, d.n), one after the other, in one CTA.
__global__ void __launch_bounds__( 1024 ) k_mg_types_dense( const __grid_constant__ SetupLevels d, int first )
{
    for( int l = first; l < d.n; ++l )
    {
        for( long long cell = threadIdx.x; cell < (long long)d.L[l].ncells; cell += blockDim.x ) dense_type( d, l, cell );
        __syncthreads();
    }
}

// Types of one dense level over the grid (levels too large for one CTA).
__global__ void k_mg_types_level( const __grid_constant__ SetupLevels d, int l )
{
    for( long long cell = blockIdx.x * (long long)blockDim.x + threadIdx.x; cell < (long long)d.L[l].ncells;
         cell += (long long)gridDim.x * blockDim.x )
        dense_type( d, l, cell );
}

// The stencil code (same bit layout as the fine code) of a fluid cell from its neighbours' types;
// wall: FluidProjection.cu:208 evaluated at the cell's lowest fine row.
__device__ __forceinline__ uint32_t stencil_code( const int* t )
{
    int diag = 6;
    uint32_t mask = 0;
#pragma unroll
    for( int q = 0; q < 6; ++q )
    {
        if( t[q] == BORA_AIR ) diag += 1;
        else if( t[q] == BORA_FLUID ) mask |= 1u << q;
        else diag -= 1;  // solid, wall, masked
    }
    return BORA_CODE_FLUID | ( (uint32_t)diag << 8 ) | mask;
}

// Codes of a tiled level with E = 4, 2 or 1 cells per tile edge, a thread per x-row.
template <int E>
__device__ __forceinline__ void codes_tiled( const SetupLevels& d, const BoraLevelDev& L, size_t row )
{
    constexpr int R = E * E, E3 = E * E * E;
    if( row >= L.ncells / E ) return;
    const int s = (int)( row / R ), y = (int)( row % E ), z = (int)( row / E % E );
    const int vt = d.tile_of[s];
    const int i0 = ( vt % d.tx ) * E, j = ( ( vt / d.tx ) % d.ty ) * E + y, k = ( vt / ( d.tx * d.ty ) ) * E + z;
    const int32_t* nb = d.nbr + (size_t)s * 27;
    // types of E cells from cell c of slot t (air in an inactive tile)
    auto types = [&]( int t, int c ) -> uint32_t {
        if( t < 0 ) return 0u;  // BORA_AIR is 0
        const uint8_t* p = L.type + (size_t)t * E3 + c;
        if constexpr( E == 4 ) return *reinterpret_cast<const uint32_t*>( p );
        else if constexpr( E == 2 ) return *reinterpret_cast<const uint16_t*>( p );
        else return *p;
    };
    const uint32_t w = types( s, E * ( y + E * z ) );
    uint32_t code[E] = {};
    bool any = false;
#pragma unroll
    for( int x = 0; x < E; ++x ) any = any || ( ( w >> ( 8 * x ) ) & 255u ) == BORA_FLUID;
    if( any )
    {
        const uint32_t ym = y > 0 ? types( s, E * ( y - 1 + E * z ) ) : types( nb[bora_dir( 0, -1, 0 )], E * ( E - 1 + E * z ) );
        const uint32_t yp = y < E - 1 ? types( s, E * ( y + 1 + E * z ) ) : types( nb[bora_dir( 0, 1, 0 )], E * ( E * z ) );
        const uint32_t zm = z > 0 ? types( s, E * ( y + E * ( z - 1 ) ) ) : types( nb[bora_dir( 0, 0, -1 )], E * ( y + E * ( E - 1 ) ) );
        const uint32_t zp = z < E - 1 ? types( s, E * ( y + E * ( z + 1 ) ) ) : types( nb[bora_dir( 0, 0, 1 )], E * y );
        const int sm = nb[bora_dir( -1, 0, 0 )], sp = nb[bora_dir( 1, 0, 0 )];
        const int xm = sm < 0 ? BORA_AIR : L.type[(size_t)sm * E3 + E * ( y + E * z ) + E - 1];
        const int xp = sp < 0 ? BORA_AIR : L.type[(size_t)sp * E3 + E * ( y + E * z )];
        const int wall = (float)( j << L.level ) + 0.5f <= d.voxel_wall + 1.f ? BORA_WALL : BORA_AIR;
        auto at = [&]( uint32_t v, int x ) { return (int)( ( v >> ( 8 * x ) ) & 255u ); };
#pragma unroll
        for( int x = 0; x < E; ++x )
        {
            if( at( w, x ) != BORA_FLUID ) continue;
            const int t[6] = { i0 + x == 0 ? wall : ( x ? at( w, x ? x - 1 : 0 ) : xm ), i0 + x + 1 >= L.nx ? wall : ( x < E - 1 ? at( w, x < E - 1 ? x + 1 : 0 ) : xp ),
                               j == 0 ? wall : at( ym, x ), j + 1 >= L.ny ? wall : at( yp, x ),
                               k == 0 ? wall : at( zm, x ), k + 1 >= L.nz ? wall : at( zp, x ) };
            code[x] = stencil_code( t );
        }
    }
    uint16_t* out = L.code + row * E;
    if constexpr( E == 4 ) *reinterpret_cast<uint2*>( out ) = make_uint2( code[0] | ( code[1] << 16 ), code[2] | ( code[3] << 16 ) );
    else if constexpr( E == 2 ) *reinterpret_cast<uint32_t*>( out ) = code[0] | ( code[1] << 16 );
    else *out = (uint16_t)code[0];
}

__device__ __forceinline__ void codes_dense( const SetupLevels& d, const BoraLevelDev& L, size_t cell )
{
    if( cell >= L.ncells ) return;
    if( L.type[cell] != BORA_FLUID ) { L.code[cell] = 0; return; }
    const int i = (int)( cell % L.dx ), j = (int)( ( cell / L.dx ) % L.dy ), k = (int)( cell / ( (size_t)L.dx * L.dy ) );
    const size_t sy = L.dx, sz = (size_t)L.dx * L.dy;
    const int wall = (float)( j << L.level ) + 0.5f <= d.voxel_wall + 1.f ? BORA_WALL : BORA_AIR;
    const int t[6] = { i == 0 ? wall : L.type[cell - 1], i + 1 >= L.nx ? wall : L.type[cell + 1],
                       j == 0 ? wall : L.type[cell - sy], j + 1 >= L.ny ? wall : L.type[cell + sy],
                       k == 0 ? wall : L.type[cell - sz], k + 1 >= L.nz ? wall : L.type[cell + sz] };
    L.code[cell] = (uint16_t)stencil_code( t );
}

// Blocks of 256 threads that level L takes in k_mg_codes.
__host__ __device__ inline size_t code_blocks( const BoraLevelDev& L )
{
    const size_t n = L.kind == 0 ? L.ncells / L.E : L.ncells;
    return ( n + 255 ) / 256;
}

// Codes of levels 1 .. d.n - 1, a level after the other in the grid.
__global__ void __launch_bounds__( 256 ) k_mg_codes( const __grid_constant__ SetupLevels d )
{
    size_t b = blockIdx.x;
    int l = 1;
    for( ; l < d.n - 1; ++l )
    {
        const size_t n = code_blocks( d.L[l] );
        if( b < n ) break;
        b -= n;
    }
    const BoraLevelDev& L = d.L[l];
    const size_t at = b * 256 + threadIdx.x;
    if( L.kind == 1 ) codes_dense( d, L, at );
    else if( L.E == 4 ) codes_tiled<4>( d, L, at );
    else if( L.E == 2 ) codes_tiled<2>( d, L, at );
    else codes_tiled<1>( d, L, at );
}

// ---- V-cycle -----------------------------------------------------------------------
//
// Navigation is specialised per level kind: tiled levels use the tile edge E as a
// compile-time constant (bit arithmetic, neighbours across tiles through the tile
// neighbour table), dense levels use their small extents. Kernels only visit the
// neighbours that the stencil code marks as fluid, which always exist.

template <int E>  // 4, 2, 1
struct TiledNav
{
    static constexpr int LE = E == 4 ? 2 : ( E == 2 ? 1 : 0 );
    static constexpr int E3 = E * E * E;
    const int32_t* nbr;
    // dense parent level (E == 1 only)
    const int32_t* tile_of;
    int tx, ty, cdx, cdy;

    __device__ inline long long nb( long long cell, int q ) const
    {
        const long long s = cell >> ( 3 * LE );
        const int l = (int)( cell & ( E3 - 1 ) );
        const int li = l & ( E - 1 ), lj = ( l >> LE ) & ( E - 1 ), lk = l >> ( 2 * LE );
        int dir, ll;
        switch( q )
        {
            case 0: if( li > 0 ) return cell - 1; dir = 12; ll = l + ( E - 1 ); break;
            case 1: if( li < E - 1 ) return cell + 1; dir = 14; ll = l - ( E - 1 ); break;
            case 2: if( lj > 0 ) return cell - E; dir = 10; ll = l + E * ( E - 1 ); break;
            case 3: if( lj < E - 1 ) return cell + E; dir = 16; ll = l - E * ( E - 1 ); break;
            case 4: if( lk > 0 ) return cell - E * E; dir = 4; ll = l + E * E * ( E - 1 ); break;
            default: if( lk < E - 1 ) return cell + E * E; dir = 22; ll = l - E * E * ( E - 1 ); break;
        }
        const int ns = nbr[s * 27 + dir];
        return ns < 0 ? -1 : (long long)ns * E3 + ll;
    }
    // parent on the next coarser level, a dense cell (E == 1: the cell is the tile)
    __device__ inline long long parent( long long cell ) const
    {
        static_assert( E == 1, "finer tiled levels run in mg_passes.cu" );
        const int vt = tile_of[cell];
        const int ti = vt % tx, tj = ( vt / tx ) % ty, tk = vt / ( tx * ty );
        return (long long)( ti >> 1 ) + (long long)cdx * ( ( tj >> 1 ) + (long long)cdy * ( tk >> 1 ) );
    }
};

struct DenseNav
{
    int dx, dy, dz;   // storage extent = cells inside the domain
    int cdx, cdy;     // coarser dense level
    __device__ inline long long nb( long long cell, int q ) const
    {
        const int c = (int)cell;  // dense levels hold far fewer than 2^31 cells
        const int i = c % dx, j = ( c / dx ) % dy, k = c / ( dx * dy );
        switch( q )
        {
            case 0: return i > 0 ? cell - 1 : -1;
            case 1: return i < dx - 1 ? cell + 1 : -1;
            case 2: return j > 0 ? cell - dx : -1;
            case 3: return j < dy - 1 ? cell + dx : -1;
            case 4: return k > 0 ? cell - (long long)dx * dy : -1;
            default: return k < dz - 1 ? cell + (long long)dx * dy : -1;
        }
    }
    __device__ inline long long parent( long long cell ) const
    {
        const int c = (int)cell;
        const int i = c % dx, j = ( c / dx ) % dy, k = c / ( dx * dy );
        return (long long)( ( i >> 1 ) + cdx * ( ( j >> 1 ) + cdy * ( k >> 1 ) ) );
    }
};

// Level residual r' of a cell (level 0 runs in mg_passes.cu).
struct RIn
{
    const __half* rh;
    __device__ inline float operator()( long long c ) const { return __half2float( rh[c] ); }
};

__device__ inline float ldh( const __half* z, long long c ) { return __half2float( z[c] ); }

// The per-level operations below are written as device functions over a strided cell
// range, so that the same code runs as one grid-wide kernel per operation (large levels)
// or, for the small tail of the hierarchy, inside one CTA that walks several levels with
// CTA barriers in between (k_mg_tail).

// z = two damped-Jacobi sweeps from zero: z1 = w r'/d, z2 = z1 + w (r' - S z1)/d, with
// each neighbour's z1 recomputed from its own r' and diagonal.
template <class Nav>
__device__ inline void smooth0_cells( const Nav& nav, const BoraLevelDev& L, const RIn& R, uint32_t* err, long long i0,
                                      long long stride )
{
    for( long long cell = i0; cell < (long long)L.ncells; cell += stride )
    {
        const uint16_t cc = L.code[cell];
        float z2 = 0.f;
        const int dg = code_diag( cc );
        if( ( cc & BORA_CODE_FLUID ) && dg > 0 )
        {
            const float rc = R( cell );
            const float z1 = kOmegaA * rc / (float)dg;
            float sum = 0.f;
#pragma unroll
            for( int q = 0; q < 6; ++q )
            {
                if( !( cc & ( 1u << q ) ) ) continue;
                const long long n = nav.nb( cell, q );
                if( n < 0 ) { atomicOr( err, 4u ); continue; }
                const int dn = code_diag( L.code[n] );
                if( dn > 0 ) sum += kOmegaA * R( n ) / (float)dn;
            }
            z2 = z1 + kOmegaB * ( rc - ( (float)dg * z1 - sum ) ) / (float)dg;
        }
        L.z0[cell] = __float2half_rn( z2 );
    }
}

// Restriction, one thread per (coarse cell, child): each thread forms its child's
// residual r' - S z (z = the pre-smoothed z0), the 8 lanes of a coarse cell add up by
// shuffles, and r'_C = 4 * mean = 0.5 * sum. C is dense; TILED: F is tiled with one cell per tile
// (children are tiles, via slot_of), else dense.
// i0 and stride are multiples of 8 apart within a warp (every lane of a warp runs the
// same number of iterations).
template <class FNav, bool TILED>
__device__ inline void restrict_cells( const FNav& fnav, const BoraLevelDev& F, const BoraLevelDev& C, const RIn& R,
                                       const int32_t* __restrict__ slot_of, int tx, int ty, int tz, uint32_t* err,
                                       long long i0, long long stride )
{
    const long long total = (long long)C.ncells * 8;
    const long long tround = ( total + 31 ) & ~31LL;
    for( long long t = i0; t < tround; t += stride )
    {
        const long long pc = t >> 3;
        const int o = (int)( t & 7 );
        float res = 0.f;
        if( t < total )  // the value of a non-fluid coarse cell is never read
        {
            long long fc = -1;
            const int I = (int)( pc % C.dx ), J = (int)( ( pc / C.dx ) % C.dy ), K = (int)( pc / ( (long long)C.dx * C.dy ) );
            const int a = 2 * I + ( o & 1 ), b = 2 * J + ( ( o >> 1 ) & 1 ), c = 2 * K + ( o >> 2 );
            if( TILED )
            {
                if( a < tx && b < ty && c < tz ) fc = slot_of[( (size_t)c * ty + b ) * tx + a];
            }
            else if( a < F.dx && b < F.dy && c < F.dz )
            {
                fc = (long long)a + (long long)F.dx * ( b + (long long)F.dy * c );
            }
            if( fc >= 0 )  // children beyond the domain are masked cells: their code is 0
            {
                const uint16_t cf = F.code[fc];
                if( cf & BORA_CODE_FLUID )
                {
                    float sum = 0.f;
#pragma unroll
                    for( int q = 0; q < 6; ++q )
                    {
                        if( !( cf & ( 1u << q ) ) ) continue;
                        const long long n = fnav.nb( fc, q );
                        if( n < 0 ) { atomicOr( err, 8u ); continue; }
                        sum += ldh( F.z0, n );
                    }
                    res = R( fc ) - ( (float)code_diag( cf ) * ldh( F.z0, fc ) - sum );
                }
            }
        }
        res += __shfl_xor_sync( 0xffffffffu, res, 1 );
        res += __shfl_xor_sync( 0xffffffffu, res, 2 );
        res += __shfl_xor_sync( 0xffffffffu, res, 4 );
        if( t < total && o == 0 ) C.r[pc] = __float2half_rn( 0.5f * res );
    }
}

// Coarsest level (<= 512 cells): Jacobi sweeps from zero in shared memory; threads 0..511
// of the CTA own one cell each, every thread of the CTA takes part in the barriers.
struct CoarsestSmem
{
    float zs[2][512], rs[512];
    int16_t nbs[512][6];
};

template <class Nav>
__device__ inline void coarsest_cells( const Nav& nav, const BoraLevelDev& L, int sweeps, uint32_t* err, CoarsestSmem& sm )
{
    const int c = threadIdx.x;
    const bool mine = c < 512;
    const bool valid = c < (int)L.ncells;
    uint16_t cc = 0;
    if( valid )
    {
        cc = L.code[c];
        sm.rs[c] = __half2float( L.r[c] );
        for( int q = 0; q < 6; ++q )
        {
            long long n = -1;
            if( cc & ( 1u << q ) )
            {
                n = nav.nb( c, q );
                if( n < 0 || n >= (long long)L.ncells ) { atomicOr( err, 16u ); n = -1; }
            }
            sm.nbs[c][q] = (int16_t)n;
        }
    }
    if( mine ) { sm.zs[0][c] = 0.f; sm.zs[1][c] = 0.f; }
    __syncthreads();
    int cur = 0;
    const int dg = code_diag( cc );
    const bool act = valid && ( cc & BORA_CODE_FLUID ) && dg > 0;
    for( int it = 0; it < sweeps; ++it )
    {
        float zn = 0.f;
        if( act )
        {
            float sum = 0.f;
            for( int q = 0; q < 6; ++q )
                if( sm.nbs[c][q] >= 0 ) sum += sm.zs[cur][sm.nbs[c][q]];
            const float z = sm.zs[cur][c];
            zn = z + kOmega * ( sm.rs[c] - ( (float)dg * z - sum ) ) / (float)dg;
        }
        if( mine ) sm.zs[cur ^ 1][c] = zn;
        __syncthreads();
        cur ^= 1;
    }
    if( valid ) L.z0[c] = __float2half_rn( sm.zs[cur][c] );
}

// z_a = z0 + P e (injection of the coarse correction C.z0), then one Jacobi sweep;
// neighbours' z_a are formed the same way. Writes z1.
template <class Nav>
__device__ inline void prolong_smooth_cells( const Nav& nav, const BoraLevelDev& F, const __half* __restrict__ ec,
                                             const RIn& R, uint32_t* err, long long i0, long long stride )
{
    for( long long cell = i0; cell < (long long)F.ncells; cell += stride )
    {
        const uint16_t cc = F.code[cell];
        float zb = 0.f;
        const int dg = code_diag( cc );
        if( ( cc & BORA_CODE_FLUID ) && dg > 0 )
        {
            const float za = ldh( F.z0, cell ) + ldh( ec, nav.parent( cell ) );
            float sum = 0.f;
#pragma unroll
            for( int q = 0; q < 6; ++q )
            {
                if( !( cc & ( 1u << q ) ) ) continue;
                const long long n = nav.nb( cell, q );
                if( n < 0 ) { atomicOr( err, 32u ); continue; }
                sum += ldh( F.z0, n ) + ldh( ec, nav.parent( n ) );
            }
            zb = za + kOmegaB * ( R( cell ) - ( (float)dg * za - sum ) ) / (float)dg;
        }
        F.z1[cell] = __float2half_rn( zb );
    }
}

// Final Jacobi sweep of a level: z = z1 + w (r' - S z1)/d, written to z0.
template <class Nav>
__device__ inline void smooth_last_cells( const Nav& nav, const BoraLevelDev& L, const RIn& R, uint32_t* err, long long i0,
                                          long long stride )
{
    for( long long cell = i0; cell < (long long)L.ncells; cell += stride )
    {
        const uint16_t cc = L.code[cell];
        float zc = 0.f;
        const int dg = code_diag( cc );
        if( ( cc & BORA_CODE_FLUID ) && dg > 0 )
        {
            const float zb = ldh( L.z1, cell );
            float sum = 0.f;
#pragma unroll
            for( int q = 0; q < 6; ++q )
            {
                if( !( cc & ( 1u << q ) ) ) continue;
                const long long n = nav.nb( cell, q );
                if( n < 0 ) { atomicOr( err, 64u ); continue; }
                sum += ldh( L.z1, n );
            }
            zc = zb + kOmegaA * ( R( cell ) - ( (float)dg * zb - sum ) ) / (float)dg;
        }
        L.z0[cell] = __float2half_rn( zc );
    }
}

// Grid-wide kernels, one per operation.
__device__ inline long long gtid() { return blockIdx.x * (long long)blockDim.x + threadIdx.x; }
__device__ inline long long gstride() { return (long long)gridDim.x * blockDim.x; }

template <class Nav>
__global__ void __launch_bounds__( 256 ) k_mg_smooth0( Nav nav, BoraLevelDev L, uint32_t* err )
{
    smooth0_cells( nav, L, RIn{ L.r }, err, gtid(), gstride() );
}

template <class FNav, bool TILED>
__global__ void __launch_bounds__( 256 ) k_mg_restrict( FNav fnav, BoraLevelDev F, BoraLevelDev C,
                                                        const int32_t* __restrict__ slot_of, int tx, int ty, int tz,
                                                        uint32_t* err )
{
    restrict_cells<FNav, TILED>( fnav, F, C, RIn{ F.r }, slot_of, tx, ty, tz, err, gtid(), gstride() );
}

template <class Nav>
__global__ void __launch_bounds__( 512 ) k_mg_coarsest( Nav nav, BoraLevelDev L, int sweeps, uint32_t* err )
{
    __shared__ CoarsestSmem sm;
    coarsest_cells( nav, L, sweeps, err, sm );
}

template <class Nav>
__global__ void __launch_bounds__( 256 ) k_mg_prolong_smooth( Nav nav, BoraLevelDev F, const __half* __restrict__ ec,
                                                              uint32_t* err )
{
    prolong_smooth_cells( nav, F, ec, RIn{ F.r }, err, gtid(), gstride() );
}

template <class Nav>
__global__ void __launch_bounds__( 256 ) k_mg_smooth_last( Nav nav, BoraLevelDev L, uint32_t* err )
{
    smooth_last_cells( nav, L, RIn{ L.r }, err, gtid(), gstride() );
}

// The small tail of the hierarchy in one thread-block cluster: levels that are dense or
// tiled with one cell per tile (only the first), down to the coarsest and back up, with a
// cluster barrier between the operations (the cluster's CTAs are co-scheduled, and the
// barrier orders their global-memory writes at cluster scope). The coarsest level runs
// in the cluster's first CTA. (Walking the levels below the first in one CTA's shared
// memory was slower: a 4096-cell level then runs on one SM.)
constexpr int kTailLevels = 8;
constexpr int kTailThreads = 1024;
constexpr int kTailCtasMax = 16;  // non-portable cluster size, where the device supports it
constexpr size_t kTailMaxCells = 32768;

__device__ inline void cluster_barrier()
{
    asm volatile( "barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory" );
}

struct TailDesc
{
    BoraLevelDev L[kTailLevels];
    int n;            // tail levels; the last is the coarsest of the hierarchy
    int first_tiled;  // L[0] is tiled with one cell per tile
    const int32_t* nbr;
    const int32_t* tile_of;
    const int32_t* slot_of;
    int tx, ty, tz;
    int sweeps;       // coarsest sweeps
};

__global__ void __launch_bounds__( kTailThreads ) k_mg_tail( const __grid_constant__ TailDesc d, uint32_t* err )
{
    __shared__ CoarsestSmem sm;
    bora_pdl_trigger();
    bora_pdl_wait();
    const long long i0 = blockIdx.x * (long long)blockDim.x + threadIdx.x, st = (long long)gridDim.x * blockDim.x;
    auto with_level = [&]( int t, auto&& f ) {
        const int cdx = t + 1 < d.n ? d.L[t + 1].dx : 0, cdy = t + 1 < d.n ? d.L[t + 1].dy : 0;
        if( t == 0 && d.first_tiled ) f( TiledNav<1>{ d.nbr, d.tile_of, d.tx, d.ty, cdx, cdy } );
        else f( DenseNav{ d.L[t].dx, d.L[t].dy, d.L[t].dz, cdx, cdy } );
    };
    for( int t = 0; t + 1 < d.n; ++t )
    {
        const RIn R{ d.L[t].r };
        with_level( t, [&]( auto nav ) { smooth0_cells( nav, d.L[t], R, err, i0, st ); } );
        cluster_barrier();
        with_level( t, [&]( auto nav ) {
            if( t == 0 && d.first_tiled )
                restrict_cells<decltype( nav ), true>( nav, d.L[t], d.L[t + 1], R, d.slot_of, d.tx, d.ty, d.tz, err, i0, st );
            else
                restrict_cells<decltype( nav ), false>( nav, d.L[t], d.L[t + 1], R, d.slot_of, d.tx, d.ty, d.tz, err, i0, st );
        } );
        cluster_barrier();
    }
    if( blockIdx.x == 0 ) with_level( d.n - 1, [&]( auto nav ) { coarsest_cells( nav, d.L[d.n - 1], d.sweeps, err, sm ); } );
    cluster_barrier();
    for( int t = d.n - 2; t >= 0; --t )
    {
        const RIn R{ d.L[t].r };
        with_level( t, [&]( auto nav ) { prolong_smooth_cells( nav, d.L[t], d.L[t + 1].z0, R, err, i0, st ); } );
        cluster_barrier();
        with_level( t, [&]( auto nav ) { smooth_last_cells( nav, d.L[t], R, err, i0, st ); } );
        cluster_barrier();
    }
}

// ---- tiled levels with E >= 2 -----------------------------------------------------------
// Levels 0, 1 and 2 (E = 8, 4, 2) run as stencil passes (mg_passes.cu).

int sm_count()
{
    static BoraPerDevice sms;
    return sms.get( [] {
        int dev = 0, n = 0;
        cudaGetDevice( &dev );
        cudaDeviceGetAttribute( &n, cudaDevAttrMultiProcessorCount, dev );
        return n > 0 ? n : 152;
    } );
}

int blocks_for( size_t n )
{
    return (int)std::max<size_t>( 1, std::min<size_t>( ( n + 255 ) / 256, (size_t)sm_count() * 8 ) );
}

}  // namespace

int bora_mg_setup( const BoraGridDev& g, BoraLevelDev* levels, int nlevels, BoraTilesDev t, void* mid_image,
                   cudaStream_t st )
{
    const int ntiles = levels[0].kind == 0 ? (int)( levels[0].ncells / 512 ) : 0;
    SetupLevels d{};
    d.n = nlevels;
    for( int l = 0; l < nlevels; ++l ) d.L[l] = levels[l];
    d.nbr = t.nbr; d.slot_of = t.slot_of; d.tile_of = t.tile_of;
    d.tx = g.tx; d.ty = g.ty; d.tz = g.tz;
    d.voxel_wall = g.voxel_wall;
    int launches = 0;
    if( nlevels < 2 ) return 0;
    k_mg_types_tiled<<<(unsigned)( ( (size_t)ntiles * 16 + 255 ) / 256 ), 256, 0, st>>>( d, ntiles );
    ++launches;
    int dense = 1;
    while( dense < nlevels && levels[dense].kind == 0 ) ++dense;
    for( ; dense < nlevels && levels[dense].ncells > kDenseOneCta; ++dense, ++launches )
        k_mg_types_level<<<blocks_for( levels[dense].ncells ), 256, 0, st>>>( d, dense );
    if( dense < nlevels )
    {
        k_mg_types_dense<<<1, 1024, 0, st>>>( d, dense );
        ++launches;
    }
    size_t blocks = 0;
    for( int l = 1; l < nlevels; ++l ) blocks += code_blocks( levels[l] );
    k_mg_codes<<<(unsigned)blocks, 256, 0, st>>>( d );
    ++launches;
    bora_mg_mid_setup( g, levels, nlevels, t, ntiles, mid_image, st );
    return launches + ( mid_image ? 1 : 0 );
}

namespace {

// Launch a level-templated kernel with the navigation of level l, dense or tiled with one cell
// per tile (the finer tiled levels run in mg_passes.cu).
template <class F>
void with_nav( const BoraGridDev& g, const BoraLevelDev* levels, int nlevels, int l, BoraTilesDev t, F&& f )
{
    const BoraLevelDev& L = levels[l];
    const int cdx = l + 1 < nlevels ? levels[l + 1].dx : 0;
    const int cdy = l + 1 < nlevels ? levels[l + 1].dy : 0;
    if( L.kind == 1 ) f( DenseNav{ L.dx, L.dy, L.dz, cdx, cdy } );
    else f( TiledNav<1>{ t.nbr, t.tile_of, g.tx, g.ty, cdx, cdy } );
}

}  // namespace

namespace {

// First level of the one-CTA tail: the longest suffix of levels that are dense (or, first
// only, tiled with one cell per tile) with at most kTailMaxCells cells; nlevels when the
// coarsest level does not qualify (tiny scenes whose coarsest level is still tiled).
int tail_start( const BoraLevelDev* levels, int nlevels )
{
    auto eligible = []( const BoraLevelDev& L ) { return L.ncells <= kTailMaxCells && ( L.kind == 1 || L.E == 1 ); };
    const int last = nlevels - 1;
    if( !eligible( levels[last] ) ) return nlevels;
    int first = last;
    while( first > 0 && eligible( levels[first - 1] ) && levels[first].kind == 1 && last - first + 2 <= kTailLevels ) --first;
    return first;
}

bool pass_level( const BoraLevelDev& L ) { return L.kind == 0 && L.E >= 2; }

// CTAs of the tail cluster: 16 where the device can co-schedule such a cluster of this
// kernel, else the portable 8.
int tail_cluster_size()
{
    static BoraPerDevice size;
    return size.get( [] {
        int n = 8;
        if( cudaFuncSetAttribute( k_mg_tail, cudaFuncAttributeNonPortableClusterSizeAllowed, 1 ) == cudaSuccess )
        {
            cudaLaunchConfig_t cfg{};
            cfg.gridDim = dim3( kTailCtasMax );
            cfg.blockDim = dim3( kTailThreads );
            cudaLaunchAttribute attr[1];
            attr[0].id = cudaLaunchAttributeClusterDimension;
            attr[0].val.clusterDim.x = kTailCtasMax;
            attr[0].val.clusterDim.y = 1;
            attr[0].val.clusterDim.z = 1;
            cfg.attrs = attr;
            cfg.numAttrs = 1;
            int clusters = 0;
            if( cudaOccupancyMaxActiveClusters( &clusters, k_mg_tail, &cfg ) == cudaSuccess && clusters > 0 ) n = kTailCtasMax;
        }
        cudaGetLastError();  // a refused query leaves no error behind
        return n;
    } );
}

}  // namespace

int bora_mg_vcycle_launches( const BoraGridDev& g, const BoraLevelDev* levels, int nlevels, BoraTilesDev t,
                             const void* mid_image )
{
    if( nlevels < 2 ) return 0;
    const int ntiles = levels[0].kind == 0 ? (int)( levels[0].ncells / 512 ) : 0;
    const int mid = bora_mg_mid_vcycle( g, levels, nlevels, t, ntiles, mid_image, nullptr, 16, nullptr, false );
    const int first = mid ? mid : tail_start( levels, nlevels );
    const int stop = std::min( first, nlevels - 1 );
    int n = 1;  // the tail kernel, or the coarsest-level kernel
    for( int l = 0; l < stop; ++l ) n += 4;
    return n;
}

void bora_mg_vcycle( const BoraGridDev& g, const BoraLevelDev* levels, int nlevels, BoraTilesDev t, BoraSolveTilesDev ft,
                     const void* mid_image, float* r, const float* q, float* z, float* scratch, BoraReduceDev red, int slot_rz_in,
                     int slot_dq_in, int slot_scale, int coarse_sweeps, cudaStream_t st )
{
    if( nlevels < 2 ) return;  // the caller always builds at least two levels
    if( levels[0].ncells == 0 ) return;
    const int last = nlevels - 1;
    const int ntiles = levels[0].kind == 0 ? (int)( levels[0].ncells / 512 ) : 0;
    // level 2 or 3 .. coarsest in one CTA or cluster out of shared memory (mg_mid.cu) when
    // the hierarchy fits it; otherwise the tail levels run from global memory (k_mg_tail)
    const int mid = bora_mg_mid_vcycle( g, levels, nlevels, t, ntiles, mid_image, red.err, coarse_sweeps, st, false );
    const int first = mid ? mid : tail_start( levels, nlevels );  // levels [first, last] run in one kernel
    const int stop = std::min( first, last );                     // levels [0, stop) restrict/prolong here
    // down: pre-smooth and restrict
    for( int l = 0; l < stop; ++l )
    {
        const BoraLevelDev& F = levels[l];
        const BoraLevelDev& C = levels[l + 1];
        if( pass_level( F ) )
        {
            bora_mg_pass_down( levels, l, ft, r, q, scratch, red, slot_scale, slot_rz_in, slot_dq_in, st );
            continue;
        }
        with_nav( g, levels, nlevels, l, t, [&]( auto nav ) {
            k_mg_smooth0<<<blocks_for( F.ncells ), 256, 0, st>>>( nav, F, red.err );
            const int nb = blocks_for( C.ncells * 8 );
            using N = decltype( nav );
            if( F.kind == 1 )
                k_mg_restrict<N, false><<<nb, 256, 0, st>>>( nav, F, C, t.slot_of, g.tx, g.ty, g.tz, red.err );
            else
                k_mg_restrict<N, true><<<nb, 256, 0, st>>>( nav, F, C, t.slot_of, g.tx, g.ty, g.tz, red.err );
        } );
    }
    if( mid )
    {
        bora_mg_mid_vcycle( g, levels, nlevels, t, ntiles, mid_image, red.err, coarse_sweeps, st, true );
    }
    else if( first <= last )
    {
        TailDesc d{};
        d.n = last - first + 1;
        for( int q = 0; q < d.n; ++q ) d.L[q] = levels[first + q];
        d.first_tiled = levels[first].kind == 0;
        d.nbr = t.nbr; d.tile_of = t.tile_of; d.slot_of = t.slot_of;
        d.tx = g.tx; d.ty = g.ty; d.tz = g.tz;
        d.sweeps = coarse_sweeps;
        const int ctas = tail_cluster_size();
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3( ctas );
        cfg.blockDim = dim3( kTailThreads );
        cfg.stream = st;
        cudaLaunchAttribute attr[2];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = ctas;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[1].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 2;
        cudaLaunchKernelEx( &cfg, k_mg_tail, d, red.err );
    }
    else
    {
        // a tiled level with four or two cells per tile's edge (a tail level would be in the tail)
        auto coarsest = [&]( auto nav ) { k_mg_coarsest<<<1, 512, 0, st>>>( nav, levels[last], coarse_sweeps, red.err ); };
        if( levels[last].E == 4 ) coarsest( TiledNav<4>{ t.nbr, t.tile_of, g.tx, g.ty, 0, 0 } );
        else coarsest( TiledNav<2>{ t.nbr, t.tile_of, g.tx, g.ty, 0, 0 } );
    }
    // up: prolong + two sweeps
    for( int l = stop - 1; l >= 0; --l )
    {
        const BoraLevelDev& F = levels[l];
        if( pass_level( F ) )
        {
            // a coarser level that ran its passes left its correction in z1, the others in z0
            const bool cf = l + 1 < stop && pass_level( levels[l + 1] );
            const __half* ec = cf ? levels[l + 1].z1 : levels[l + 1].z0;
            bora_mg_pass_up( levels, l, ec, ft, r, scratch, red, slot_scale, z, st );
            continue;
        }
        with_nav( g, levels, nlevels, l, t, [&]( auto nav ) {
            k_mg_prolong_smooth<<<blocks_for( F.ncells ), 256, 0, st>>>( nav, F, levels[l + 1].z0, red.err );
            k_mg_smooth_last<<<blocks_for( F.ncells ), 256, 0, st>>>( nav, F, red.err );
        } );
    }
}

void bora_member_grids( int nft, int* grid, const int* v )
{
    bora_projection_grids( nft, grid );
    grid[kGridPass0] = bora_mg_pass_grid( 8, nft, v[0] );
    grid[kGridPass0R] = bora_mg_pass_grid( 8, nft, -1 );
    grid[kGridPass1] = bora_mg_pass_grid( 4, nft, v[1] );
    grid[kGridPass2] = bora_mg_pass_grid( 2, nft, v[2] );
}
