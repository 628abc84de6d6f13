// G2P with the FLIP/PIC blend, Euler advection substeps with the box clamp and collider
// push-out, kill flags and gravity: FLIPMethod::updateParticles
// (base/source/FLIPMethod.cu:54-175), followed by the compaction of Array::remove
// (base/header/Array.h:996-1024, FLIPMethod.cu:293-297).
//
// Particles are visited in dual-cell order through the sort permutation and written
// to the other particle buffer in that order, so the particle store stays spatially
// sorted and each warp's trilinear reads hit the same few cells. Killed particles are
// written with id -1 and dropped by the next step's counting sort. Each written particle
// is also binned for the next rebuild (its sort key and tile flag, the rule of k_bin), so
// that the next step need not read the particles again to bin them; a tile's CTA marks the
// flags of the 27 tiles around its own in shared memory and stores each marked one once.
#include <algorithm>

#include "bora_internal.h"
#include "../../include/bora_flip.h"

namespace {

// Grid values of a tile and its high-side halo layer, (8+1)^3 cells, staged in shared memory: a
// float4 (comp.x, comp.y, velo.x, velo.y) and a float2 (comp.z, velo.z) per cell, so that the
// lerps of both vector fields take two loads per corner, and per base cell surf's minimum over
// the eight corners. Cells of inactive tiles hold the field backgrounds (0, and 10 for surf:
// FLIPMethod.cu:30).
constexpr int kG2PThreads = 256;
constexpr int kG2PSplitMax = 4;  // CTAs per tile at most
constexpr int kStageEdge = BORA_TILE + 1;
constexpr int kStageCells = kStageEdge * kStageEdge * kStageEdge;

// SparseField::lerp over a vector field (base/header/SparseField.h:150-173) and
// SparseField::lerpMin over a scalar field (SparseField.h:176-196), from the staged tile.
// Corner order: (i,j,k),(i+1,j,k),(i,j,k+1),(i+1,j,k+1),(i,j+1,k),(i+1,j+1,k),(i,j+1,k+1),
// (i+1,j+1,k+1).
struct StagedLerp
{
    int base;  // staged index of corner (i,j,k)
    int cell;  // its index in the tile
    bool staged;  // the base cell lies in the tile
    float x, y, z;
    __device__ inline void setup( const BoraGridDev& g, int ti, int tj, int tk, float px, float py, float pz )
    {
        const int i = bora_clampi( bora_trunc( px - 0.5f ), 0, g.nx - 2 );
        const int j = bora_clampi( bora_trunc( py - 0.5f ), 0, g.ny - 2 );
        const int k = bora_clampi( bora_trunc( pz - 0.5f ), 0, g.nz - 2 );
        x = bora_clampf( px - ( (float)i + .5f ), 0.f, 1.f );
        y = bora_clampf( py - ( (float)j + .5f ), 0.f, 1.f );
        z = bora_clampf( pz - ( (float)k + .5f ), 0.f, 1.f );
        // (for the particles of the tile's dual cells it does: the frame's extent is a multiple of
        // 4, so that the clamp above leaves i in the tile)
        const int li = i - ti * BORA_TILE, lj = j - tj * BORA_TILE, lk = k - tk * BORA_TILE;
        base = li + kStageEdge * ( lj + kStageEdge * lk );
        cell = li + BORA_TILE * ( lj + BORA_TILE * lk );
        staged = ( (unsigned)li | (unsigned)lj | (unsigned)lk ) < (unsigned)BORA_TILE;
    }
    __device__ static inline int off( int q )
    {
        return ( q & 1 ) + kStageEdge * kStageEdge * ( ( q >> 1 ) & 1 ) + kStageEdge * ( q >> 2 );
    }
    __device__ static inline float4 mix( float4 a, float4 b, float t )
    {
        return make_float4( a.x * ( 1.f - t ) + b.x * t, a.y * ( 1.f - t ) + b.y * t, a.z * ( 1.f - t ) + b.z * t,
                            a.w * ( 1.f - t ) + b.w * t );
    }
    // the same by packed pairs: two FP32 operations an instruction, each rounded as alone. The sum
    // is a fused b t * one + a (1 - t) with one = 1 from memory, because the compiler would fuse
    // a packed product into a packed sum, which rounds once.
    __device__ static inline float2 mix( float2 a, float2 b, float t, float one )
    {
        return __ffma2_rn( __fmul2_rn( b, make_float2( t, t ) ), make_float2( one, one ),
                           __fmul2_rn( a, make_float2( 1.f - t, 1.f - t ) ) );
    }
    __device__ static inline float4 mix( float4 a, float4 b, float t, float one )
    {
        const float2 lo = mix( make_float2( a.x, a.y ), make_float2( b.x, b.y ), t, one );
        const float2 hi = mix( make_float2( a.z, a.w ), make_float2( b.z, b.w ), t, one );
        return make_float4( lo.x, lo.y, hi.x, hi.y );
    }
    __device__ static inline float fminf_ref( float a, float b ) { return a < b ? a : b; }  // MathUtils.h:174
    // the minimum of surf over the corners of the base cell at staged index b, in SparseField's order
    __device__ static inline float corner_min( const float* surf, int b )
    {
        auto w = [&]( int q ) { return surf[b + off( q )]; };
        float v = fminf_ref( w( 0 ), w( 1 ) );
        v = fminf_ref( v, fminf_ref( w( 2 ), w( 3 ) ) );
        v = fminf_ref( v, fminf_ref( w( 4 ), w( 5 ) ) );
        return fminf_ref( v, fminf_ref( w( 6 ), w( 7 ) ) );
    }
    // comp alone
    __device__ inline float4 comp( const float4* fa, const float2* fb, float one ) const
    {
        auto xy = [&]( int q ) { return *reinterpret_cast<const float2*>( fa + base + off( q ) ); };
        auto cz = [&]( int q ) { return make_float2( fb[base + off( q )].x, 0.f ); };
        auto lerp = [&]( auto f ) {
            const float2 c00 = mix( f( 0 ), f( 1 ), x, one ), c01 = mix( f( 2 ), f( 3 ), x, one );
            const float2 c10 = mix( f( 4 ), f( 5 ), x, one ), c11 = mix( f( 6 ), f( 7 ), x, one );
            return mix( mix( c00, c10, y, one ), mix( c01, c11, y, one ), z, one );
        };
        const float2 a = lerp( xy ), b = lerp( cz );
        return make_float4( a.x, a.y, b.x, 0.f );
    }
    // comp and velo lerped from the staged cells (comp.xy and velo.xy from fa, comp.z and
    // velo.z from fb); the corners' mix order is SparseField's
    __device__ inline void sample( const float4* fa, const float2* fb, float one, float4& comp, float4& velo ) const
    {
        auto lerp = [&]( const auto* f ) {
            const auto c00 = mix( f[base + off( 0 )], f[base + off( 1 )], x, one );
            const auto c01 = mix( f[base + off( 2 )], f[base + off( 3 )], x, one );
            const auto c10 = mix( f[base + off( 4 )], f[base + off( 5 )], x, one );
            const auto c11 = mix( f[base + off( 6 )], f[base + off( 7 )], x, one );
            return mix( mix( c00, c10, y, one ), mix( c01, c11, y, one ), z, one );
        };
        const float4 A = lerp( fa );
        const float2 B = lerp( fb );
        comp = make_float4( A.x, A.y, B.x, 0.f );
        velo = make_float4( A.z, A.w, B.y, 0.f );
    }
};

// The same lerps through the tile table, for the rare particles outside every tile (the
// sort's last bin: particles added outside the grid, killed by this step's bounds check).
struct GlobalLerp
{
    const BoraGridDev& g;
    const int32_t* slot_of;
    const BoraCellsDev& c;
    int idx[8];  // cell index, -1 = background (inactive tile)
    float x, y, z;
    __device__ inline int index( int i, int j, int k ) const
    {
        const int s = slot_of[( (size_t)( k >> 3 ) * g.ty + ( j >> 3 ) ) * g.tx + ( i >> 3 )];
        return s < 0 ? -1 : s * BORA_TILE_CELLS + bora_local( i, j, k );
    }
    __device__ inline void setup( float px, float py, float pz )
    {
        const int i = bora_clampi( bora_trunc( px - 0.5f ), 0, g.nx - 2 );
        const int j = bora_clampi( bora_trunc( py - 0.5f ), 0, g.ny - 2 );
        const int k = bora_clampi( bora_trunc( pz - 0.5f ), 0, g.nz - 2 );
        x = bora_clampf( px - ( (float)i + .5f ), 0.f, 1.f );
        y = bora_clampf( py - ( (float)j + .5f ), 0.f, 1.f );
        z = bora_clampf( pz - ( (float)k + .5f ), 0.f, 1.f );
        for( int q = 0; q < 8; ++q ) idx[q] = index( i + ( q & 1 ), j + ( q >> 2 ), k + ( ( q >> 1 ) & 1 ) );
    }
    __device__ inline float4 fa( int q ) const
    {
        return idx[q] < 0 ? make_float4( 0.f, 0.f, 0.f, 10.f )
                          : make_float4( c.cx[idx[q]], c.cy[idx[q]], c.cz[idx[q]], c.surf[idx[q]] );
    }
    __device__ inline float4 fb( int q ) const
    {
        return idx[q] < 0 ? make_float4( 0.f, 0.f, 0.f, 0.f ) : make_float4( c.vx[idx[q]], c.vy[idx[q]], c.vz[idx[q]], 0.f );
    }
    template <bool A>
    __device__ inline float4 lerp() const
    {
        auto f = [&]( int q ) { return A ? fa( q ) : fb( q ); };
        const float4 c00 = StagedLerp::mix( f( 0 ), f( 1 ), x );
        const float4 c01 = StagedLerp::mix( f( 2 ), f( 3 ), x );
        const float4 c10 = StagedLerp::mix( f( 4 ), f( 5 ), x );
        const float4 c11 = StagedLerp::mix( f( 6 ), f( 7 ), x );
        return StagedLerp::mix( StagedLerp::mix( c00, c10, y ), StagedLerp::mix( c01, c11, y ), z );
    }
    __device__ inline float surf_min() const
    {
        auto w = [&]( int q ) { return fa( q ).w; };
        float v = StagedLerp::fminf_ref( w( 0 ), w( 1 ) );
        v = StagedLerp::fminf_ref( v, StagedLerp::fminf_ref( w( 2 ), w( 3 ) ) );
        v = StagedLerp::fminf_ref( v, StagedLerp::fminf_ref( w( 4 ), w( 5 ) ) );
        v = StagedLerp::fminf_ref( v, StagedLerp::fminf_ref( w( 6 ), w( 7 ) ) );
        return v;
    }
    __device__ inline float4 comp() const { return lerp<true>(); }
    __device__ inline float4 velo() const { return lerp<false>(); }
};

__device__ inline bool inside_grid( const BoraGridDev& g, float x, float y, float z )
{
    return !( x < 0.f || x > (float)g.nx || y < 0.f || y > (float)g.ny || z < 0.f || z > (float)g.nz );
}

// Collider interactions of FLIPMethod::updateParticles, kept out of line: they are rare,
// and their corner arrays would otherwise spill the common path's registers.
__device__ __noinline__ float3 col_carry( const BoraGridDev* g, float3 p, float dt )
{
    if( bora_col_phi( *g, p.x, p.y, p.z ) < 0.f )  // FLIPMethod.cu:116-119
    {
        float cv[3];
        bora_col_lerp( g->cols, g->nx, g->ny, g->nz, p.x, p.y, p.z, 2, cv );
        p.x += cv[0] * dt; p.y += cv[1] * dt; p.z += cv[2] * dt;
    }
    return p;
}

// push-out along the collider normal (FLIPMethod.cu:146-157); w = 1 when it collided
__device__ __noinline__ float4 col_push( const BoraGridDev* g, float3 p )
{
    const float phi = bora_col_phi( *g, p.x, p.y, p.z );
    if( !( phi < 0.f ) ) return make_float4( p.x, p.y, p.z, 0.f );
    float nr[3];
    bora_col_lerp( g->cols, g->nx, g->ny, g->nz, p.x, p.y, p.z, 1, nr );
    // Vec3f::normalized (base/header/Vector3.h:350-354)
    const double dn = 1.0f / sqrtf( nr[0] * nr[0] + nr[1] * nr[1] + nr[2] * nr[2] + 1e-30f );
    const float ux = (float)( nr[0] * dn ), uy = (float)( nr[1] * dn ), uz = (float)( nr[2] * dn );
    return make_float4( p.x - ux * phi, p.y - uy * phi, p.z - uz * phi, 1.f );
}

__device__ __noinline__ bool col_kill( const BoraGridDev* g, float3 p )
{
    const float phi = bora_col_phi( *g, p.x, p.y, p.z );  // FLIPMethod.cu:161-165
    return phi > 3.f || phi < 0.f;
}

// The CTA's staged tile, for lookups away from the particle's own position (fa null: none).
struct StagedTile
{
    const float4* fa;
    const float2* fb;
    float one;
    int ti, tj, tk;
};

// Grid velocity ("comp") at an arbitrary point, for the RK2 option: from the staged tile where the
// point's base cell lies in it, else through the tile table.
__device__ inline float4 comp_at( const BoraGridDev& g, const int32_t* slot_of, const BoraCellsDev& c, const StagedTile& st,
                                  float x, float y, float z )
{
    if( st.fa )
    {
        StagedLerp l;
        l.setup( g, st.ti, st.tj, st.tk, x, y, z );
        if( l.staged ) return l.comp( st.fa, st.fb, st.one );
    }
    GlobalLerp l{ g, slot_of, c };
    l.setup( x, y, z );
    return l.comp();
}

// FLIPMethod::updateParticles for one particle (FLIPMethod.cu:60-170); gn and go are the
// grid's projected and pre-projection velocities lerped at the particle's position. With the
// RK2 option each substep moves the particle by the midpoint rule in the grid velocity field
// instead of by its own velocity; everything else is unchanged. The modes compile the common case
// alone (no water tank, no colliders, Euler advection), the water tank and the colliders with Euler
// advection, and everything (the caller checks). kCols = false leaves a particle that may meet a
// collider alone and returns kLater: the collider code's calls would spill the registers of the
// others. sub[]: dt / iter for 0 < iter < kSubTable.
enum AdvanceMode { kCommon, kEuler, kEverything };
constexpr int kSubTable = 32;
constexpr int kLater = 2;

template <int kMode, bool kCols>
__device__ inline int advance_particle( const BoraGridDev& g, float4 gn, float4 go, const int32_t* slot_of,
                                         const BoraCellsDev& c, float& px, float& py, float& pz, float& vx, float& vy,
                                         float& vz, float dt, const float* sub, const StagedTile& st )
{
    constexpr bool kAll = kMode != kCommon, kRk2 = kMode == kEverything;
    const float lx = (float)g.nx + 0.5f, lz = (float)g.nz + 0.5f;
    const float wall = g.voxel_wall;
    {
        vx += gn.x - go.x; vy += gn.y - go.y; vz += gn.z - go.z;
        vx = vx * 0.95f + gn.x * 0.05f;
        vy = vy * 0.95f + gn.y * 0.05f;
        vz = vz * 0.95f + gn.z * 0.05f;
    }
    if( kAll && g.enable_tank && py <= wall )
    {
        const float band = g.damping_band;
        float w = 1.f;
        if( px < band ) w = fminf( w, bora_clampf( ( px - 0.f ) / band, 0.f, 1.f ) );
        if( px > lx - band ) w = fminf( w, bora_clampf( ( lx - px ) / band, 0.f, 1.f ) );
        if( pz < band ) w = fminf( w, bora_clampf( ( pz - 0.f ) / band, 0.f, 1.f ) );
        if( pz > lz - band ) w = fminf( w, bora_clampf( ( lz - pz ) / band, 0.f, 1.f ) );
        vx *= w; vy *= w; vz *= w;
    }
    // Collider work only where a collider can be met this step: the substep positions stay
    // within |v| dt of the start (the box clamp only shortens moves of particles that start
    // inside the grid), a sampled collider value is a lerp of box distances at cell centres
    // within sqrt(3) cells, and a box distance changes by at most the distance moved. So a
    // particle whose start is farther than 2 |v| dt + 2 cells from every box sees positive
    // collider values all step long. (RK2 moves with the grid velocity: no cull.)
    bool hasCols = kAll && bora_col_active( g.cols );
    if( hasCols && g.cols.tslot && !( kRk2 && g.advection == BORA_ADVECT_RK2 ) && inside_grid( g, px, py, pz ) )
    {
        // sparse collider: every sample outside its tiles is the (positive) background with
        // a zero normal and velocity; a particle whose tile has no collider tile within one
        // tile is 8 cells or more from every stored sample, and the samples it reads this
        // step lie within |v| dt + 3 cells of its start
        const float move = sqrtf( vx * vx + vy * vy + vz * vz ) * dt;
        if( g.cols.tbg > 0.f && move < 5.f )
        {
            const int ti = bora_imin( bora_trunc( px ) >> 3, g.tx - 1 ), tj = bora_imin( bora_trunc( py ) >> 3, g.ty - 1 ),
                      tk = bora_imin( bora_trunc( pz ) >> 3, g.tz - 1 );
            if( !g.cols.tnear[(size_t)ti + (size_t)g.tx * ( (size_t)tj + (size_t)g.ty * tk )] ) hasCols = false;
        }
    }
    else if( hasCols && !g.cols.fphi && !( kRk2 && g.advection == BORA_ADVECT_RK2 ) && inside_grid( g, px, py, pz ) )
    {
        const float reach = 2.f * sqrtf( vx * vx + vy * vy + vz * vz ) * dt + 2.f;
        hasCols = false;
        for( int n = 0; n < g.cols.count; ++n )
            if( !( bora_box_sdf( g.cols.box[n], px, py, pz ) > reach ) ) hasCols = true;
    }
    if( !kCols && hasCols ) return kLater;
    if( kCols && hasCols )
    {
        const float3 p = col_carry( &g, make_float3( px, py, pz ), dt );
        px = p.x; py = p.y; pz = p.z;
    }
    bool kill = false;
    {
        const float len = sqrtf( vx * vx + vy * vy + vz * vz );
        const int iter = 1 + bora_imin( bora_trunc( len * dt * 1.5f ), bora_imax( g.maxsubsteps, 1 ) );
        // (iter is 0 or negative for a negative dt: the loop does not run, and the table is not read)
        const float sub_dt = (unsigned)iter < (unsigned)kSubTable ? sub[iter] : dt / (float)iter;
        bool col = false;
        for( int it = 0; it < iter; ++it )
        {
            if( kRk2 && g.advection == BORA_ADVECT_RK2 )
            {
                const float h = 0.5f * sub_dt;
                // the first substep starts where gn was sampled, unless a collider carried the particle
                const float4 k1 = it == 0 && !( kCols && hasCols ) ? gn : comp_at( g, slot_of, c, st, px, py, pz );
                const float4 k2 = comp_at( g, slot_of, c, st, px + k1.x * h, py + k1.y * h, pz + k1.z * h );
                px += k2.x * sub_dt; py += k2.y * sub_dt; pz += k2.z * sub_dt;
            }
            else
            {
                px += vx * sub_dt; py += vy * sub_dt; pz += vz * sub_dt;
            }
            if( py <= wall )
            {
                if( px < 0.f ) { px = 0.f; if( vx < 0.f ) vx = 0.f; }
                if( py < 0.f ) { py = 0.f; if( vy < 0.f ) vy = 0.f; }
                if( pz < 0.f ) { pz = 0.f; if( vz < 0.f ) vz = 0.f; }
                if( px > (float)g.nx ) { px = (float)g.nx; if( vx > 0.f ) vx = 0.f; }
                if( py > (float)g.ny ) { py = (float)g.ny; if( vy > 0.f ) vy = 0.f; }
                if( pz > (float)g.nz ) { pz = (float)g.nz; if( vz > 0.f ) vz = 0.f; }
            }
            if( kCols && hasCols )
            {
                const float4 r = col_push( &g, make_float3( px, py, pz ) );
                px = r.x; py = r.y; pz = r.z;
                if( r.w != 0.f ) col = true;
            }
        }
        if( kCols && col && col_kill( &g, make_float3( px, py, pz ) ) ) kill = true;
        if( !inside_grid( g, px, py, pz ) ) kill = true;
    }
    vx += g.gravity[0] * dt; vy += g.gravity[1] * dt; vz += g.gravity[2] * dt;
    return kill ? 1 : 0;
}

// Mark of a particle left for the collider loop (no key: those are below the dead keys).
constexpr uint32_t kLaterKey = BORA_DEAD_KEY - 2;

// One CTA per tile: stage the tile's grid values, then advance the particles of the
// tile's dual cells (a contiguous range of the sorted order). The CTA after the last tile
// advances the sort's outside bin through the tile table.
//
// Bound by the particles' gathers through L1 and by instructions: at 256^3 (24.6 M particles, 8.2
// K tiles) 435 us in 500 instructions a particle at 80 registers (three CTAs per SM), 384
// at 64 (four): lerps by packed pairs, surf's minimum once per base cell instead of per particle,
// dt / iter from a table, the sort key of a particle that is known to be inside the grid. A 640
// tank with a collider 1097 -> 817, its collider calls in a loop of their own, whose
// spills the others do not pay for; an RK2 step at 96^3 134 -> 113 at 80 registers (119
// at 64), and 82 with its lookups from the staged tile instead of through the tile table, the
// first one being the sample that the particle already has.
template <int kMode>
__global__ void __launch_bounds__( kG2PThreads, kMode == kEverything ? 3 : 4 ) k_g2p( const __grid_constant__ BoraGridDev g, BoraTilesDev t, int ntiles,
                                                       uint32_t nsorted, const uint32_t* __restrict__ start, BoraCellsDev c,
                                                       BoraParticlesDev src, const uint32_t* __restrict__ idx,
                                                       BoraParticlesDev dst, float* __restrict__ adj, float dt,
                                                       uint32_t* __restrict__ nkilled, uint32_t* vkey,
                                                       uint8_t* __restrict__ tile_flag )
{
    __shared__ float4 fa[kStageCells];  // comp.x, comp.y, velo.x, velo.y
    __shared__ float2 fb[kStageCells];  // comp.z, velo.z
    __shared__ float surf[kStageCells], surf_min[BORA_TILE_CELLS];
    __shared__ int32_t nb[27];
    __shared__ uint8_t near_flag[27];  // activation flags of the tiles around the CTA's own
    __shared__ float sub[kSubTable];   // dt / iter; [0] is 1
    const int s = blockIdx.x, tid = threadIdx.x;
    // a tile's CTAs (grid y) take its particles in turns
    const uint32_t first = blockIdx.y * kG2PThreads + tid, stride = gridDim.y * kG2PThreads;
    if( tid < kSubTable ) sub[tid] = tid ? dt / (float)tid : 1.f;
    uint32_t kills = 0;
    int cti = -8, ctj = -8, ctk = -8;  // the CTA's tile (far from every tile: no shared flags)
    auto finish = [&]( uint32_t q, uint32_t pi, int32_t id, float px, float py, float pz, float vx, float vy, float vz,
                       bool kill ) {
        dst.px[q] = px; dst.py[q] = py; dst.pz[q] = pz;
        dst.vx[q] = vx; dst.vy[q] = vy; dst.vz[q] = vz;
        dst.id[q] = kill ? -1 : id;
        uint32_t key = BORA_DEAD_KEY;
        if( !kill && id >= 0 )
        {
            // (a particle that lives is inside the grid)
            int ti, tj, tk;
            bora_bin_tile_inside( g.tx, g.ty, g.tz, px, py, pz, ti, tj, tk );
            const int dx = ti - cti, dy = tj - ctj, dz = tk - ctk;
            if( dx >= -1 && dx <= 1 && dy >= -1 && dy <= 1 && dz >= -1 && dz <= 1 ) near_flag[bora_dir( dx, dy, dz )] = 1;
            else tile_flag[( (size_t)tk * g.ty + tj ) * g.tx + ti] = 1;
            key = bora_bin_inside_key( g.tx, g.ty, px, py, pz );
        }
        vkey[q] = key;
        if( dst.vort )  // post-processing attributes ride along (FLIPMethod.cu:295-296)
        {
            dst.vort[q] = src.vort[pi];
            dst.curv[q] = src.curv[pi];
        }
        kills += kill ? 1u : 0u;
    };
    if( s == ntiles )
    {
        __syncthreads();
        const uint32_t q0 = start[(size_t)ntiles * BORA_TILE_CELLS], q1 = nsorted;
        for( uint32_t q = q0 + first; q < q1; q += stride )
        {
            const uint32_t pi = idx[q];
            float px = src.px[pi], py = src.py[pi], pz = src.pz[pi];
            float vx = src.vx[pi], vy = src.vy[pi], vz = src.vz[pi];
            GlobalLerp smp{ g, t.slot_of, c };
            smp.setup( px, py, pz );
            adj[q] = smp.surf_min();
            const int kill = advance_particle<kMode, true>( g, smp.comp(), smp.velo(), t.slot_of, c, px, py, pz, vx, vy, vz, dt, sub,
                                                               StagedTile{} );
            finish( q, pi, src.id[pi], px, py, pz, vx, vy, vz, kill != 0 );
        }
    }
    else
    {
        if( tid < 27 ) nb[tid] = t.nbr[(size_t)s * 27 + tid];
        if( tid < 27 ) near_flag[tid] = 0;
        const int vt = t.tile_of[s];
        const int ti = vt % g.tx, tj = ( vt / g.tx ) % g.ty, tk = vt / ( g.tx * g.ty );
        cti = ti; ctj = tj; ctk = tk;
        // the thread's particles are loaded one ahead and their sorted-order indices two ahead:
        // the first particle and the second index before the staging, then each next particle
        // (from an index that has arrived) while the current one is advanced
        const uint32_t q0 = start[(size_t)s * BORA_TILE_CELLS], q1 = start[(size_t)( s + 1 ) * BORA_TILE_CELLS];
        uint32_t pin = 0, pin2 = 0;
        int32_t idn = 0;
        float pxn = 0.f, pyn = 0.f, pzn = 0.f, vxn = 0.f, vyn = 0.f, vzn = 0.f;
        auto fetch = [&]( uint32_t pi ) {
            pxn = src.px[pi]; pyn = src.py[pi]; pzn = src.pz[pi];
            vxn = src.vx[pi]; vyn = src.vy[pi]; vzn = src.vz[pi];
            idn = src.id[pi];
        };
        if( q0 + first < q1 )
        {
            pin = idx[q0 + first];
            fetch( pin );
        }
        if( q0 + first + stride < q1 ) pin2 = idx[q0 + first + stride];
        __syncthreads();
        for( int h = tid; h < kStageCells; h += kG2PThreads )
        {
            const int a = h % kStageEdge, b = ( h / kStageEdge ) % kStageEdge, cz = h / ( kStageEdge * kStageEdge );
            const int ns = nb[bora_dir( a >> 3, b >> 3, cz >> 3 )];
            float4 va = make_float4( 0.f, 0.f, 0.f, 0.f );
            float2 vb = make_float2( 0.f, 0.f );
            float vs = 10.f;
            if( ns >= 0 )
            {
                const size_t q = (size_t)ns * BORA_TILE_CELLS + (size_t)bora_local( a, b, cz );
                va = make_float4( c.cx[q], c.cy[q], c.vx[q], c.vy[q] );
                vb = make_float2( c.cz[q], c.vz[q] );
                vs = c.surf[q];
            }
            fa[h] = va;
            fb[h] = vb;
            surf[h] = vs;
        }
        __syncthreads();
        for( int l = tid; l < BORA_TILE_CELLS; l += kG2PThreads )
            surf_min[l] = StagedLerp::corner_min( surf, ( l & 7 ) + kStageEdge * ( ( ( l >> 3 ) & 7 ) + kStageEdge * ( l >> 6 ) ) );
        __syncthreads();
        const StagedTile st{ fa, fb, sub[0], ti, tj, tk };
        uint32_t later = 0;  // particles of this thread that wait for the collider code
        for( uint32_t q = q0 + first; q < q1; q += stride )
        {
            const uint32_t pi = pin;
            const int32_t id = idn;
            float px = pxn, py = pyn, pz = pzn;
            float vx = vxn, vy = vyn, vz = vzn;
            if( q + stride < q1 )
            {
                pin = pin2;
                fetch( pin );
                if( q + 2 * stride < q1 ) pin2 = idx[q + 2 * stride];
            }
            StagedLerp l;
            l.setup( g, ti, tj, tk, px, py, pz );
            float4 gn, go;
            l.sample( fa, fb, sub[0], gn, go );
            adj[q] = surf_min[l.cell];
            const int kill = advance_particle<kMode, false>( g, gn, go, t.slot_of, c, px, py, pz, vx, vy, vz, dt, sub, st );
            if( kMode != kCommon && kill == kLater )
            {
                vkey[q] = kLaterKey;
                ++later;
                continue;
            }
            finish( q, pi, id, px, py, pz, vx, vy, vz, kill != 0 );
        }
        if constexpr( kMode != kCommon )
#pragma unroll 1
            for( uint32_t q = q0 + first; later != 0 && q < q1; q += stride )
            {
                if( vkey[q] != kLaterKey ) continue;
                --later;
                const uint32_t pi = idx[q];
                float px = src.px[pi], py = src.py[pi], pz = src.pz[pi];
                float vx = src.vx[pi], vy = src.vy[pi], vz = src.vz[pi];
                StagedLerp l;
                l.setup( g, ti, tj, tk, px, py, pz );
                float4 gn, go;
                l.sample( fa, fb, sub[0], gn, go );
                const int kill = advance_particle<kMode, true>( g, gn, go, t.slot_of, c, px, py, pz, vx, vy, vz, dt, sub, st );
                finish( q, pi, src.id[pi], px, py, pz, vx, vy, vz, kill != 0 );
            }
        __syncthreads();
        if( tid < 27 && near_flag[tid] )  // a marked tile is a clamped particle tile: inside the table
        {
            const int i = cti + tid % 3 - 1, j = ctj + ( tid / 3 ) % 3 - 1, k = ctk + tid / 9 - 1;
            tile_flag[( (size_t)k * g.ty + j ) * g.tx + i] = 1;
        }
    }
    // one atomic per warp
    for( int o = 16; o > 0; o >>= 1 ) kills += __shfl_xor_sync( 0xffffffffu, kills, o );
    if( ( threadIdx.x & 31 ) == 0 && kills ) atomicAdd( nkilled, kills );
}

}  // namespace

void bora_launch_g2p( const BoraGridDev& g, int ntiles, size_t nsorted, BoraTilesDev t, const uint32_t* start, BoraCellsDev c,
                      BoraParticlesDev src, const uint32_t* idx, BoraParticlesDev dst, float* adj, float dt,
                      uint32_t* nkilled, uint32_t* vkey, uint8_t* tile_flag, cudaStream_t st )
{
    if( nsorted == 0 ) return;
    // Few tiles: up to four CTAs each, so that two rounds of the chip's 608 places are taken (a tile's
    // particles are a chain of 16 rounds in one CTA): 26 us at 24^3 (27 tiles) and 30 at 64^3 (240)
    // with one, 14 and 22 with four; at 360 tiles 25 with one, 23 with three; at 432, 504 and 576
    // tiles 31, 33 and 35 with one, 27, 28 and 31 with two; one from 608 tiles on.
    const int split = std::max( 1, std::min( kG2PSplitMax, 1216 / ( ntiles + 1 ) ) );
    // the common case in a kernel without the code of the others, and the RK2 lookups (two more
    // grid samples, inlined) only where they are asked for
    auto go = [&]( auto kernel ) {
        kernel<<<dim3( ntiles + 1, split ), kG2PThreads, 0, st>>>( g, t, ntiles, (uint32_t)nsorted, start, c, src, idx, dst, adj, dt,
                                                    nkilled, vkey, tile_flag );
    };
    if( g.advection == BORA_ADVECT_RK2 ) go( k_g2p<kEverything> );
    else if( g.enable_tank || bora_col_active( g.cols ) ) go( k_g2p<kEuler> );
    else go( k_g2p<kCommon> );
}
