// Sparse field -> VDB conversion on the device, as 8^3 leaf blocks.
//
// The Houdini node turns the surface and velocity fields into OpenVDB grids after every
// frame (houdini/source/SOP_FlipWater.cpp:252-264) with FieldCast's convertSurfaceVDB
// (base/header/FieldCast.h:362-440) and convertVelocityVDB (:14-48). OpenVDB's leaf nodes
// are 8^3 voxel blocks at multiples of 8, exactly the frame's tiles (VDB voxel (i,j,k) =
// frame cell (i,j,k), transform: voxel size dx, translate min + dx/2), so the conversion
// here writes one leaf per tile - origin, 512-bit active mask and 512 values - and a caller
// that has OpenVDB copies leaves straight into a tree:
//   surface:  value = phi * dx over the cells of active tiles inside the grid (active),
//             background * dx elsewhere (inactive); with the water tank on, every voxel of
//             the 3-cell border band (below the grid, and around its sides up to 3 cells
//             above the water level) becomes active with min(cell centre y - level, value)
//             (FieldCast.h:398-440), which adds the leaves of the band outside the tiles;
//   velocity: value = v * dx (Grid::worldVector) over the cells of active tiles inside the
//             grid, active unless |v| < 1e-30 (FieldCast.h:33-45), 0 elsewhere.
// The float arithmetic follows FieldCast's operation order (this unit is compiled without
// floating-point contraction).
#include <algorithm>
#include <vector>

#include "bora_internal.h"

namespace {

struct VdbBand
{
    int on;            // water tank
    int ei, ek;        // last cell index per axis (grid nx - 1, nz - 1)
    int lv;            // int( (level - min.y) / dx + 1 )
    float level;       // water level (world)
    float ty, sy;      // world transform in y: y = j' * sy + ty for voxel coordinate j'
};

// FieldCast.h:408-438: the five slabs of the band (3 cells wide)
__device__ inline bool in_band( const VdbBand& b, int i, int j, int k )
{
    constexpr int bnd = 3;
    const bool ik_all = i >= -bnd && i <= b.ei + bnd && k >= -bnd && k <= b.ek + bnd;
    if( !ik_all || j < -bnd ) return false;
    if( j <= 0 ) return true;                  // below / at the grid bottom
    if( j > b.lv + bnd ) return false;
    return i <= 0 || i >= b.ei || k <= 0 || k >= b.ek;  // the four side walls
}

__global__ void k_vdb_leaves( BoraGridDev g, int ntiles, const int32_t* __restrict__ tile_of, int4* __restrict__ leaf )
{
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if( s >= ntiles ) return;
    const int vt = tile_of[s];
    leaf[s] = make_int4( 8 * ( vt % g.tx ), 8 * ( ( vt / g.tx ) % g.ty ), 8 * ( vt / ( g.tx * g.ty ) ), s );
}

// One CTA per leaf, one thread per voxel (x fastest). The leaf's flag (any voxel active), or its
// origin, mask and values at its place among the kept leaves: a leaf is written once, packed, so
// that the caller's arrays are filled by three copies (one copy per leaf took 22 ms for the
// surface and velocity of 1398 tiles).
__device__ __forceinline__ void vdb_emit( const BoraVdbOut& o, int q, const int4& lf, bool act )
{
    const int l = threadIdx.x;
    if( o.flag )
    {
        const int any = __syncthreads_or( act );
        if( l == 0 ) o.flag[q] = any ? 1 : 0;
        return;
    }
    const unsigned bits = __ballot_sync( 0xffffffffu, act );
    if( ( l & 31 ) == 0 ) reinterpret_cast<uint32_t*>( o.mask + (size_t)q * 8 )[l >> 5] = bits;
    if( l < 3 ) o.origin[3 * (size_t)q + l] = l == 0 ? lf.x : ( l == 1 ? lf.y : lf.z );
}

__global__ void __launch_bounds__( 512 ) k_vdb_surface( int nx, int ny, int nz, BoraVdbOut o, const float* __restrict__ surf,
                                                        float dx, float bg, VdbBand band )
{
    const int q = blockIdx.x, l = threadIdx.x;
    const int4 lf = o.leaf[o.keep ? o.keep[q] : q];
    const int i = lf.x + ( l & 7 ), j = lf.y + ( ( l >> 3 ) & 7 ), k = lf.z + ( l >> 6 );
    float v = bg * dx;
    bool act = false;
    if( lf.w >= 0 && i >= 0 && j >= 0 && k >= 0 && i < nx && j < ny && k < nz )
    {
        if( !o.flag ) v = surf[(size_t)lf.w * BORA_TILE_CELLS + l] * dx;
        act = true;
    }
    if( band.on && in_band( band, i, j, k ) )
    {
        const float cy = ( (float)j + 0.5f ) * band.sy + band.ty;  // Grid::worldPoint
        const float a = cy - band.level;
        v = a < v ? a : v;  // Min
        act = true;
    }
    if( !o.flag ) o.val[(size_t)q * 512 + l] = v;
    vdb_emit( o, q, lf, act );
}

__global__ void __launch_bounds__( 512 ) k_vdb_velocity( int nx, int ny, int nz, BoraVdbOut o, const float* __restrict__ vx,
                                                         const float* __restrict__ vy, const float* __restrict__ vz,
                                                         float3 scale )
{
    const int q = blockIdx.x, l = threadIdx.x;
    const int4 lf = o.leaf[o.keep ? o.keep[q] : q];
    const int i = lf.x + ( l & 7 ), j = lf.y + ( ( l >> 3 ) & 7 ), k = lf.z + ( l >> 6 );
    float wx = 0.f, wy = 0.f, wz = 0.f;
    bool act = false;
    if( lf.w >= 0 && i < nx && j < ny && k < nz )
    {
        const size_t c = (size_t)lf.w * BORA_TILE_CELLS + l;
        wx = vx[c] * scale.x;  // Grid::worldVector
        wy = vy[c] * scale.y;
        wz = vz[c] * scale.z;
        act = !( sqrtf( wx * wx + wy * wy + wz * wz ) < 1e-30f );  // Vec3f::length
        if( !act ) wx = wy = wz = 0.f;
    }
    if( !o.flag )
    {
        float* d = o.val + ( (size_t)q * 512 + l ) * 3;
        d[0] = wx;
        d[1] = wy;
        d[2] = wz;
    }
    vdb_emit( o, q, lf, act );
}

// Four cells per thread: three 16-byte reads and three 16-byte writes.
__global__ void k_interleave( size_t n4, const float4* __restrict__ x, const float4* __restrict__ y, const float4* __restrict__ z,
                              float4* __restrict__ out )
{
    for( size_t v = blockIdx.x * (size_t)blockDim.x + threadIdx.x; v < n4; v += (size_t)gridDim.x * blockDim.x )
    {
        const float4 a = x[v], b = y[v], c = z[v];
        out[3 * v] = make_float4( a.x, b.x, c.x, a.y );
        out[3 * v + 1] = make_float4( b.y, c.y, a.z, b.z );
        out[3 * v + 2] = make_float4( c.z, a.w, b.w, c.w );
    }
}

__global__ void k_deinterleave( size_t n4, const float4* __restrict__ in, float4* __restrict__ x, float4* __restrict__ y,
                                float4* __restrict__ z )
{
    for( size_t v = blockIdx.x * (size_t)blockDim.x + threadIdx.x; v < n4; v += (size_t)gridDim.x * blockDim.x )
    {
        const float4 a = in[3 * v], b = in[3 * v + 1], c = in[3 * v + 2];
        x[v] = make_float4( a.x, a.w, b.z, c.y );
        y[v] = make_float4( a.y, b.x, b.w, c.z );
        z[v] = make_float4( a.z, b.y, c.x, c.w );
    }
}

int blocks_for_quads( size_t n4 ) { return (int)std::max<size_t>( 1, std::min<size_t>( ( n4 + 255 ) / 256, 152 * 16 ) ); }

}  // namespace

// FieldCast.h:404, int lv = (waterlevel - min.y) / dx + 1, with the float kept inside int range
int bora_vdb_level_index( float level, float min_y, float dx )
{
    const float f = ( level - min_y ) / dx + 1.f;
    return (int)std::max( -1.0e9f, std::min( 1.0e9f, f ) );
}

void bora_launch_vdb_leaves( const BoraGridDev& g, int ntiles, const int32_t* tile_of, int4* leaf, cudaStream_t st )
{
    if( ntiles > 0 ) k_vdb_leaves<<<( ntiles + 255 ) / 256, 256, 0, st>>>( g, ntiles, tile_of, leaf );
}

void bora_launch_vdb_surface( const BoraGridDev& g, const float* scale, const float* translate, const BoraVdbOut& o,
                              const float* surf, float bg, int tank, float level, cudaStream_t st )
{
    if( o.n <= 0 ) return;
    const float dx = scale[0];
    VdbBand b{};
    b.on = tank;
    b.ei = g.nx - 1;
    b.ek = g.nz - 1;
    b.lv = bora_vdb_level_index( level, translate[1], dx );
    b.level = level;
    b.ty = translate[1];
    b.sy = scale[1];
    k_vdb_surface<<<o.n, 512, 0, st>>>( g.nx, g.ny, g.nz, o, surf, dx, bg, b );
}

void bora_launch_vdb_velocity( const BoraGridDev& g, const float* scale, const BoraVdbOut& o, const float* vx, const float* vy,
                               const float* vz, cudaStream_t st )
{
    if( o.n <= 0 ) return;
    k_vdb_velocity<<<o.n, 512, 0, st>>>( g.nx, g.ny, g.nz, o, vx, vy, vz, make_float3( scale[0], scale[1], scale[2] ) );
}

void bora_launch_interleave( size_t n, const float* x, const float* y, const float* z, float* out, cudaStream_t st )
{
    if( n )
        k_interleave<<<blocks_for_quads( n / 4 ), 256, 0, st>>>( n / 4, (const float4*)x, (const float4*)y, (const float4*)z, (float4*)out );
}

void bora_launch_deinterleave( size_t n, const float* in, float* x, float* y, float* z, cudaStream_t st )
{
    if( n )
        k_deinterleave<<<blocks_for_quads( n / 4 ), 256, 0, st>>>( n / 4, (const float4*)in, (float4*)x, (float4*)y, (float4*)z );
}

// The band's leaves (tile coordinates, possibly -1 or one past the tile grid) for the
// water tank with level `level`: every tile that holds a voxel of the band.
void bora_vdb_band_tiles( const BoraGridDev& g, const float* scale, const float* translate, float level,
                          std::vector<int32_t>& tiles )
{
    const float dx = scale[0];
    const int ei = g.nx - 1, ek = g.nz - 1;
    const int lv = bora_vdb_level_index( level, translate[1], dx );
    constexpr int bnd = 3;
    auto tile_of = []( int c ) { return c >= 0 ? c / 8 : -( ( -c + 7 ) / 8 ); };
    const int ti0 = tile_of( -bnd ), ti1 = tile_of( ei + bnd ), tk0 = tile_of( -bnd ), tk1 = tile_of( ek + bnd );
    const int tj0 = tile_of( -bnd ), tj1 = tile_of( std::max( 0, lv + bnd ) );
    for( int tk = tk0; tk <= tk1; ++tk )
        for( int tj = tj0; tj <= tj1; ++tj )
            for( int ti = ti0; ti <= ti1; ++ti )
            {
                // does the tile hold a band voxel? (the band is a union of boxes)
                const int i0 = ti * 8, j0 = tj * 8, k0 = tk * 8;
                const int i1 = i0 + 7, j1 = j0 + 7, k1 = k0 + 7;
                auto overlap = [&]( int a0, int a1, int b0, int b1 ) { return a0 <= b1 && b0 <= a1; };
                const bool ik = overlap( i0, i1, -bnd, ei + bnd ) && overlap( k0, k1, -bnd, ek + bnd );
                if( !ik ) continue;
                bool hit = overlap( j0, j1, -bnd, 0 );
                if( !hit && overlap( j0, j1, -bnd, lv + bnd ) )
                    hit = overlap( i0, i1, -bnd, 0 ) || overlap( i0, i1, ei, ei + bnd ) || overlap( k0, k1, -bnd, 0 ) ||
                          overlap( k0, k1, ek, ek + bnd );
                if( hit )
                {
                    tiles.push_back( ti );
                    tiles.push_back( tj );
                    tiles.push_back( tk );
                }
            }
}
