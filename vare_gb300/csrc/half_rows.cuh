#pragma once

#include "bora_internal.h"

__device__ inline void tile_coords( const BoraGridDev& g, int vt, int& ti, int& tj, int& tk )
{
    ti = vt % g.tx;
    tj = ( vt / g.tx ) % g.ty;
    tk = vt / ( g.tx * g.ty );
}

// Stencils over the active tiles outside the solve, one warp per half tile (z layers 0..3 or
// 4..7), a lane per x-row (lane = j + 8 (k mod 4)), as the solve's kernels walk theirs. Cells of
// inactive tiles and beyond the grid read as air and zero.

struct HalfRow
{
    bool mine;              // past the last half tile: nothing is stored, every neighbour is inactive
    int s, hi;              // the tile's slot; the half
    int xm, xp, yt, zt;     // slots at the row's x ends; of the rows that no other lane holds (-1: none)
    int c, yc, zc;          // cells of the row, and of those rows, in their tiles
    int j, kk;              // the lane's row in the half
    int i0, J, K;           // the row's first cell in the grid
    __device__ size_t at() const { return (size_t)s * BORA_TILE_CELLS + c; }
};

// W: half tiles (warps) per CTA
template <int W>
__device__ __forceinline__ HalfRow half_row( const BoraGridDev& g, const BoraTilesDev& t, int ntiles )
{
    HalfRow r;
    const int lane = threadIdx.x & 31, h = (int)blockIdx.x * W + (int)( threadIdx.x >> 5 );
    r.mine = h < 2 * ntiles;
    r.s = r.mine ? h >> 1 : 0;
    r.hi = h & 1;
    r.j = lane & 7;
    r.kk = lane >> 3;
    r.c = r.hi * 256 + 8 * lane;
    const int32_t* nb = t.nbr + (size_t)r.s * 27;
    auto slot = [&]( int d ) { return r.mine ? __ldg( nb + d ) : -1; };
    r.xm = slot( bora_dir( -1, 0, 0 ) );
    r.xp = slot( bora_dir( 1, 0, 0 ) );
    const int ym = slot( bora_dir( 0, -1, 0 ) ), yp = slot( bora_dir( 0, 1, 0 ) ), z = slot( bora_dir( 0, 0, r.hi ? 1 : -1 ) );
    const int own = r.mine ? r.s : -1;
    r.yt = r.j == 0 ? ym : ( r.j == 7 ? yp : -1 );
    r.yc = r.c + ( r.j == 0 ? 56 : -56 );
    r.zt = r.kk == 0 ? ( r.hi ? own : z ) : ( r.kk == 3 ? ( r.hi ? z : own ) : -1 );
    r.zc = 8 * r.j + ( r.kk == 0 ? ( r.hi ? 192 : 448 ) : ( r.hi ? 0 : 256 ) );
    int ti, tj, tk;
    tile_coords( g, t.tile_of[r.s], ti, tj, tk );
    r.i0 = ti * BORA_TILE;
    r.J = tj * BORA_TILE + r.j;
    r.K = tk * BORA_TILE + 4 * r.hi + r.kk;
    return r;
}

// 8 values of a row (`background` in an inactive tile)
__device__ __forceinline__ void row8( const float* __restrict__ f, int t, int c, float* v, float background = 0.f )
{
#pragma unroll
    for( int i = 0; i < 8; ++i ) v[i] = background;
    if( t >= 0 ) bora_ld8( f + (size_t)t * BORA_TILE_CELLS + c, v );
}

// the values of a field next to a row in y or z: from the other lanes, or the loaded row
__device__ __forceinline__ void beside( const float* v, const float* halo, int step, bool first, bool last, float* m, float* p )
{
    const int lane = threadIdx.x & 31;
#pragma unroll
    for( int i = 0; i < 8; ++i )
    {
        const float a = __shfl_sync( 0xffffffffu, v[i], lane - step ), b = __shfl_sync( 0xffffffffu, v[i], lane + step );
        m[i] = first ? halo[i] : a;
        p[i] = last ? halo[i] : b;
    }
}

// CTAs for the half tiles of ntiles tiles
inline int row_grid( int ntiles, int W ) { return ( 2 * ntiles + W - 1 ) / W; }
