// The coarse tail of the multigrid V-cycle (level 3, one cell per 8^3 tile, down to the
// coarsest level and back; level 2 alone where it is the coarsest) in one thread-block cluster whose CTAs keep every value in
// distributed shared memory.
//
// Levels 0-2 are large and run as grid-wide stencil passes (mg_passes.cu). Below them
// the hierarchy is tiny (level 3 has one cell per active tile, then dense grids halved per
// level down to <= 512 cells). Run from global memory every operation of these levels is a
// chain of dependent global loads (tile tables, codes, neighbours' values) followed by a
// cluster barrier: 3-7 us per operation, 43 us per V-cycle at 256^3 for 12.5 K cells. Here
// the cluster's CTAs split every level by ownership (contiguous slot ranges of level 3,
// contiguous index ranges of the dense levels, the coarsest level in CTA 0). Everything
// that is static during a solve - stencil codes and, per owned cell, packed references
// (owning CTA, local index) of its six face neighbours, its parent and its eight children -
// is laid out once per step by k_mg_mid_image as one block per CTA in global memory, in the
// CTA's shared-memory layout, and each V-cycle copies its block in with asynchronous
// 16-byte copies before waiting for the previous kernel. The operations then run out of
// shared memory: a CTA reads other cells' values from the owning CTA's shared memory
// through the cluster window and writes only its own.
//
// An operation is one chain of latencies (references, values, store, barrier), so its loads
// are issued together, without a branch on the neighbour or its owner: 1200-1600 cycles
// instead of 2400-4400 with one dependent load after another. At 256^3 (9.4 K level-3 cells)
// the kernel takes 33 K cycles instead of 52 K, at 96^3 (726 cells, one CTA) 15 K instead of
// 29 K; a whole V-cycle there went from 137 to 128 us and from 57 to 48 us.
//
// The arithmetic is the V-cycle of multigrid.cu: per level two Jacobi sweeps before
// (kOmegaA from zero, then kOmegaB) and after (kOmegaB, then kOmegaA), the residual
// restricted as 0.5 * sum of the 8 children, injection as prolongation, and damped Jacobi
// sweeps from zero on the coarsest level; values stay FP32 inside the kernel (the grid-
// wide kernels store FP16 between launches). Operations of a level, each followed by a
// cluster barrier:
//   down:  B = z after the second pre-smoothing sweep (A holds the first, pointwise sweep)
//          A = residual r - S B
//          r, A of the coarser level = 0.5 * sum of the children's A, its pointwise sweep
//   up:    A = B + Z(parent)      (Z: the coarser level's final correction)
//          B = A + wB (r - S A)
//          A = B + wA (r - S B)   (the level's final correction)
// Non-fluid cells hold 0 in A and B and are never summed (the stencil code's neighbour
// bits select the fluid neighbours).
#include <algorithm>
#include <cooperative_groups.h>
#include <cstring>

#include <cuda_fp16.h>

#include "bora_internal.h"

namespace cg = cooperative_groups;

namespace {

constexpr float kOmega = 0.9f;      // coarsest level: damped Jacobi
constexpr float kOmegaA = 0.5687f;  // Chebyshev pair of the smoothers (multigrid.cu)
constexpr float kOmegaB = 1.6902f;

// Threads per CTA: one per level-3 cell within these bounds (a cluster barrier costs 611
// cycles with 256 threads a CTA and 924 with 1024, whatever the cluster's size).
constexpr int kMidThreadsMin = 256, kMidThreadsMax = 1024;
// Level-3 cells up to which one CTA runs the levels, with its own barrier and loads, instead
// of a cluster of 16. Cycles from the level-2 residual on: 12.3 K against 16.3 K at 726
// cells, 15.6 K against 19.7 K at 1526, but 24.0 K against 22.4 K at 2568.
constexpr int kMidSingleMax = 2048;
constexpr int kMidMaxLevels = 8;
constexpr int kMidCtasMax = 16;  // non-portable cluster size where the device allows it
constexpr size_t kMidSmemMax = 200 * 1024 + 512;

// A packed reference to a cell: owning CTA in bits 24-31, local index in bits 0-23. Every
// value array has one more entry than the CTA has cells, which stays 0: a reference that
// names no cell points there, so an operation issues all of its loads at once.
__device__ inline int32_t pack_ref( int owner, int local ) { return ( owner << 24 ) | local; }

struct MidLevel
{
    int E;           // cells per tile edge: 2 (level 2, the coarsest), 1 (level 3); 0: dense
    int n;           // cells
    int chunk;       // cells per CTA (the coarsest level: all, in CTA 0)
    int dx, dy, dz;  // dense extent
    const uint16_t* code;                          // global stencil codes (static during a solve)
    int o_code, o_nb, o_par, o_ch;                 // static block: byte offsets (-1: none)
    int o_r, o_a, o_b;                             // values: byte offsets after the static block
};

struct MidDesc
{
    MidLevel L[kMidMaxLevels];
    int n;  // levels; L[0] is level 2 or 3 of the hierarchy; the last is the coarsest
    const int32_t* nbr;
    const int32_t* tile_of;
    const int32_t* slot_of;
    int tx, ty, tz;
    const __half* r_in;  // the first level's residual (written by the finer level's down kernel)
    __half* z_out;       // its correction (read by the finer level's up kernel)
    int sweeps;
    int ctas, threads;
    int static_bytes;    // bytes of a CTA's static block (a multiple of 16)
    char* image;         // ctas static blocks, built by k_mg_mid_image
    uint32_t* err;       // inconsistent stencil codes are recorded here
};

extern __shared__ __align__( 16 ) char g_mid_smem[];

// In the image: the code names a fluid neighbour that does not exist. Recorded in d.err when
// the V-cycle first loads the cell's code; the neighbour counts as 0.
constexpr uint16_t kCodeBad = 0x4000;

__device__ inline int code_diag( uint16_t c ) { return ( c >> 8 ) & 15; }

// face directions in the 27-entry tile neighbour table: -x +x -y +y -z +z
__device__ __constant__ int kFaceDir[6] = { 12, 14, 10, 16, 4, 22 };

// ONE: the cluster is one CTA.
template <bool ONE>
struct Mid
{
    const MidDesc& d;
    cg::cluster_group cl;
    unsigned me;

    template <class T> __device__ T* arr( int off ) const { return reinterpret_cast<T*>( g_mid_smem + off ); }
    __device__ int owned( const MidLevel& L ) const
    {
        const int lo = (int)me * L.chunk;
        return L.n > lo ? min( L.chunk, L.n - lo ) : 0;
    }
    __device__ int32_t ref( const MidLevel& L, int c ) const  // packed reference of cell c of L
    {
        const int o = c / L.chunk;
        return pack_ref( o, c - o * L.chunk );
    }
    __device__ int32_t zero_ref( const MidLevel& L ) const { return pack_ref( (int)me, L.chunk ); }
    // the value at a packed reference in array `off`, from the owning CTA's shared memory
    // (volatile: stays between the barriers; no branch on the owner, so that the loads of
    // an operation are in flight together)
    __device__ float ld( int off, int32_t rf ) const
    {
        if( ONE ) return arr<float>( off )[rf & 0xFFFFFF];
        const uint32_t sa = (uint32_t)__cvta_generic_to_shared( g_mid_smem ) + (uint32_t)off + (uint32_t)( rf & 0xFFFFFF ) * 4u;
        uint32_t ra;
        float v;
        asm volatile( "mapa.shared::cluster.u32 %0, %1, %2;" : "=r"( ra ) : "r"( sa ), "r"( (uint32_t)rf >> 24 ) );
        asm volatile( "ld.shared::cluster.f32 %0, [%1];" : "=f"( v ) : "r"( ra ) );
        return v;
    }
    __device__ void barrier() const
    {
        if( ONE ) __syncthreads();
        else cl.sync();
    }

    // cell of level L next to cell c in direction q (-x +x -y +y -z +z), or -1
    __device__ int neighbour( const MidLevel& L, int c, int q ) const
    {
        const int s = q & 1 ? 1 : -1, ax = q >> 1;
        if( L.E )
        {
            const int sh = L.E == 2 ? 1 : 0, l = c & ( L.E * L.E * L.E - 1 ), bit = 1 << ax;
            const int t = c >> ( 3 * sh );
            const int at = sh ? ( l >> ax ) & 1 : 0;  // the cell's coordinate on the axis inside its tile
            const int l2 = sh ? l ^ bit : l;          // one cell along the axis, in this tile or wrapped into the next
            if( at + s >= 0 && at + s < L.E ) return ( t << ( 3 * sh ) ) | l2;
            const int tn = d.nbr[(size_t)t * 27 + kFaceDir[q]];
            return tn < 0 ? -1 : ( tn << ( 3 * sh ) ) | l2;
        }
        const int x = c % L.dx, y = ( c / L.dx ) % L.dy, z = c / ( L.dx * L.dy );
        const int at = ax == 0 ? x : ( ax == 1 ? y : z ), n = ax == 0 ? L.dx : ( ax == 1 ? L.dy : L.dz );
        if( at + s < 0 || at + s >= n ) return -1;
        return c + s * ( ax == 0 ? 1 : ( ax == 1 ? L.dx : L.dx * L.dy ) );
    }
    // static data of level t for the owned cells (codes, neighbours, parent, children),
    // written into the block at `blk` (the CTA's slice of the image) by `parts` CTAs
    __device__ void stage( int t, char* blk, int part, int parts ) const
    {
        const MidLevel& L = d.L[t];
        const int n = owned( L ), base = (int)me * L.chunk;
        const int i0 = part * (int)blockDim.x + (int)threadIdx.x, di = parts * (int)blockDim.x;
        uint16_t* code = reinterpret_cast<uint16_t*>( blk + L.o_code );
        int32_t* nb = reinterpret_cast<int32_t*>( blk + L.o_nb );
        for( int i = i0; i < n; i += di )
        {
            const int c = base + i;
            uint16_t cc = L.code[c], bad = 0;
#pragma unroll
            for( int q = 0; q < 6; ++q )
            {
                const int nc = neighbour( L, c, q );
                const bool on = ( cc & BORA_CODE_FLUID ) && ( cc & ( 1u << q ) );
                if( on && nc < 0 ) bad = kCodeBad;
                nb[q * L.chunk + i] = on && nc >= 0 ? ref( L, nc ) : zero_ref( L );
            }
            code[i] = cc | bad;
        }
        if( L.o_par >= 0 )
        {
            const MidLevel& P = d.L[t + 1];
            int32_t* par = reinterpret_cast<int32_t*>( blk + L.o_par );
            for( int i = i0; i < n; i += di )
            {
                const int c = base + i;
                int x, y, z;
                if( L.E )
                {
                    const int vt = d.tile_of[c];
                    x = vt % d.tx; y = ( vt / d.tx ) % d.ty; z = vt / ( d.tx * d.ty );
                }
                else
                {
                    x = c % L.dx; y = ( c / L.dx ) % L.dy; z = c / ( L.dx * L.dy );
                }
                par[i] = ref( P, ( x >> 1 ) + P.dx * ( ( y >> 1 ) + P.dy * ( z >> 1 ) ) );
            }
        }
        if( L.o_ch >= 0 )
        {
            const MidLevel& F = d.L[t - 1];
            int32_t* ch = reinterpret_cast<int32_t*>( blk + L.o_ch );
            for( int i = i0; i < n * 8; i += di )
            {
                const int lc = i / 8, o = i % 8, c = base + lc;
                const int x = c % L.dx, y = ( c / L.dx ) % L.dy, z = c / ( L.dx * L.dy );
                const int a = 2 * x + ( o & 1 ), b = 2 * y + ( ( o >> 1 ) & 1 ), e = 2 * z + ( o >> 2 );
                int fc = -1;
                if( F.E )
                {
                    if( a < d.tx && b < d.ty && e < d.tz ) fc = d.slot_of[( (size_t)e * d.ty + b ) * d.tx + a];
                }
                else if( a < F.dx && b < F.dy && e < F.dz )
                {
                    fc = a + F.dx * ( b + F.dy * e );
                }
                ch[o * L.chunk + lc] = fc >= 0 ? ref( F, fc ) : zero_ref( F );
            }
        }
    }

    // r - S z at an owned cell, from its own value and its fluid neighbours' in array `in`
    __device__ float defect( const MidLevel& L, int lc, uint16_t cc, int in, float z ) const
    {
        const int32_t* nb = arr<int32_t>( L.o_nb ) + lc;
        int32_t rf[6];
        float v[6];
#pragma unroll
        for( int q = 0; q < 6; ++q ) rf[q] = nb[q * L.chunk];
#pragma unroll
        for( int q = 0; q < 6; ++q ) v[q] = ld( in, rf[q] );
        const float sum = ( ( ( ( v[0] + v[1] ) + v[2] ) + v[3] ) + v[4] ) + v[5];
        return arr<float>( L.o_r )[lc] - ( (float)code_diag( cc ) * z - sum );
    }
    // store( cell, in + w[d] (r - S in) ) on the owned fluid cells, 0 elsewhere
    template <class Store>
    __device__ void sweep( int t, int in, const float* w, Store store ) const
    {
        const MidLevel& L = d.L[t];
        const int n = owned( L );
        for( int lc = threadIdx.x; lc < n; lc += (int)blockDim.x )
        {
            const uint16_t cc = arr<uint16_t>( L.o_code )[lc];
            const int dg = code_diag( cc );
            const float z = arr<float>( in )[lc];
            const float e = defect( L, lc, cc, in, z );
            store( lc, ( cc & BORA_CODE_FLUID ) && dg > 0 ? z + w[dg] * e : 0.f );
        }
    }
    // A = r - S B on the owned cells (0 on non-fluid cells)
    __device__ void residual( int t ) const
    {
        const MidLevel& L = d.L[t];
        const int n = owned( L );
        float* res = arr<float>( L.o_a );
        for( int lc = threadIdx.x; lc < n; lc += (int)blockDim.x )
        {
            const uint16_t cc = arr<uint16_t>( L.o_code )[lc];
            const float e = defect( L, lc, cc, L.o_b, arr<float>( L.o_b )[lc] );
            res[lc] = ( cc & BORA_CODE_FLUID ) ? e : 0.f;
        }
    }
    // level t (>= 1): r = 0.5 * sum of the children's residuals (A of level t - 1), and the
    // first pre-smoothing sweep from zero, A = w[d] r
    __device__ void gather( int t, const float* w ) const
    {
        const MidLevel& L = d.L[t];
        const int fa = d.L[t - 1].o_a;
        const int n = owned( L );
        for( int lc = threadIdx.x; lc < n; lc += (int)blockDim.x )
        {
            const int32_t* ch = arr<int32_t>( L.o_ch ) + lc;
            int32_t rf[8];
            float v[8];
#pragma unroll
            for( int o = 0; o < 8; ++o ) rf[o] = ch[o * L.chunk];
#pragma unroll
            for( int o = 0; o < 8; ++o ) v[o] = ld( fa, rf[o] );
            const float s0 = ( ( v[0] + v[2] ) + v[4] ) + v[6], s1 = ( ( v[1] + v[3] ) + v[5] ) + v[7];
            const float rv = 0.5f * ( s0 + s1 );
            const uint16_t cc = arr<uint16_t>( L.o_code )[lc];
            const int dg = code_diag( cc );
            if( cc & kCodeBad ) atomicOr( d.err, 4u );
            arr<float>( L.o_r )[lc] = rv;
            arr<float>( L.o_a )[lc] = ( ( cc & BORA_CODE_FLUID ) && dg > 0 ) ? w[dg] * rv : 0.f;
        }
    }
    // A = B + Z(parent) on the owned fluid cells (Z = array zoff of level t + 1)
    __device__ void inject( int t, int zoff ) const
    {
        const MidLevel& L = d.L[t];
        const int n = owned( L );
        for( int lc = threadIdx.x; lc < n; lc += (int)blockDim.x )
        {
            const uint16_t cc = arr<uint16_t>( L.o_code )[lc];
            const float z = arr<float>( L.o_b )[lc] + ld( zoff, arr<int32_t>( L.o_par )[lc] );
            arr<float>( L.o_a )[lc] = ( cc & BORA_CODE_FLUID ) && code_diag( cc ) > 0 ? z : 0.f;
        }
    }
    // The coarsest level's sweeps from the second on, A to B to A. A thread keeps its K
    // cells' weights, residuals and neighbours' offsets in registers, and the warps that
    // hold cells meet at a barrier of their own. 16 sweeps of 16 barriers: latency, so the
    // loop has explicit shared-memory accesses and no branch (107 cycles a sweep at 125
    // cells and 190 at 512, against 214 and 264 with pointers picked per sweep).
    template <int K>
    __device__ __forceinline__ void coarsest( const MidLevel& L, int sweeps, const float* w ) const
    {
        const int T = ( ( L.n + K - 1 ) / K + 31 ) / 32 * 32;  // threads that hold cells
        const int tid = (int)threadIdx.x;
        if( tid >= T ) return;
        const uint32_t sa = (uint32_t)__cvta_generic_to_shared( g_mid_smem );
        const uint32_t A = sa + (uint32_t)L.o_a, B = sa + (uint32_t)L.o_b;
        uint32_t nb[K][6], own[K];
        float z[K], rc[K], wd[K], fd[K];
        bool mine[K], act[K];
#pragma unroll
        for( int k = 0; k < K; ++k )
        {
            const int c = tid + k * T;
            mine[k] = c < L.n;
            own[k] = 4u * (uint32_t)( mine[k] ? c : L.n );
            const uint16_t cc = mine[k] ? arr<uint16_t>( L.o_code )[c] : (uint16_t)0;
            act[k] = ( cc & BORA_CODE_FLUID ) && code_diag( cc ) > 0;
            wd[k] = w[code_diag( cc )];
            fd[k] = (float)code_diag( cc );
            rc[k] = mine[k] ? arr<float>( L.o_r )[c] : 0.f;
            z[k] = mine[k] ? arr<float>( L.o_a )[c] : 0.f;
#pragma unroll
            for( int q = 0; q < 6; ++q )  // owner 0: the index is local
                nb[k][q] = mine[k] ? 4u * (uint32_t)( arr<int32_t>( L.o_nb )[q * L.chunk + c] & 0xFFFFFF ) : 4u * (uint32_t)L.n;
        }
        auto step = [&]( uint32_t in, uint32_t out ) {
            float v[K][6];
#pragma unroll
            for( int k = 0; k < K; ++k )
#pragma unroll
                for( int q = 0; q < 6; ++q ) asm volatile( "ld.shared.f32 %0, [%1];" : "=f"( v[k][q] ) : "r"( in + nb[k][q] ) );
#pragma unroll
            for( int k = 0; k < K; ++k )
            {
                const float sum = ( ( ( ( v[k][0] + v[k][1] ) + v[k][2] ) + v[k][3] ) + v[k][4] ) + v[k][5];
                z[k] = act[k] ? z[k] + wd[k] * ( rc[k] - ( fd[k] * z[k] - sum ) ) : 0.f;
                if( mine[k] ) asm volatile( "st.shared.f32 [%0], %1;" ::"r"( out + own[k] ), "f"( z[k] ) : "memory" );
            }
            asm volatile( "bar.sync 1, %0;" ::"r"( T ) : "memory" );
        };
        for( int it = 1; it < sweeps; it += 2 )
        {
            step( A, B );
            if( it + 1 < sweeps ) step( B, A );
        }
    }
};

// kImageParts CTAs per cluster CTA: lay out that CTA's static block of the image (once per step).
constexpr int kImageParts = 8;
__global__ void __launch_bounds__( 256 ) k_mg_mid_image( const __grid_constant__ MidDesc d )
{
    Mid<false> m{ d, cg::this_cluster(), blockIdx.x / kImageParts };
    char* blk = d.image + (size_t)m.me * d.static_bytes;
    for( int t = 0; t < d.n; ++t ) m.stage( t, blk, (int)( blockIdx.x % kImageParts ), kImageParts );
}

template <bool ONE>
__device__ __forceinline__ void mg_mid_body( const MidDesc& d )
{
    __shared__ float wA[16], wB[16], wC[16];
    Mid<ONE> m{ d, cg::this_cluster(), 0u };
    if( !ONE ) m.me = m.cl.block_rank();
    const int tid = threadIdx.x;
    bora_pdl_trigger();
    if( tid < 16 )
    {
        wA[tid] = tid ? kOmegaA / (float)tid : 0.f;
        wB[tid] = tid ? kOmegaB / (float)tid : 0.f;
        wC[tid] = tid ? kOmega / (float)tid : 0.f;
    }
    // the static block (no kernel of the solve writes it) before the dependency wait:
    // asynchronous 16-byte copies, all in flight at once
    {
        const char* src = d.image + (size_t)m.me * d.static_bytes;
        const uint32_t dst = (uint32_t)__cvta_generic_to_shared( g_mid_smem );
        for( int i = tid * 16; i < d.static_bytes; i += (int)blockDim.x * 16 )
            asm volatile( "cp.async.cg.shared.global [%0], [%1], 16;" ::"r"( dst + i ), "l"( src + i ) : "memory" );
        asm volatile( "cp.async.commit_group;" ::: "memory" );
    }
    // the entry behind each value array that unused references read
    if( tid < d.n * 2 )
    {
        const MidLevel& L = d.L[tid >> 1];
        m.template arr<float>( tid & 1 ? L.o_b : L.o_a )[L.chunk] = 0.f;
    }
    bora_pdl_wait();  // the finer level's restricted residual is complete from here
    const int last = d.n - 1;
    {
        const MidLevel& L = d.L[0];
        const int n = m.owned( L );
        const uint16_t* code = m.template arr<uint16_t>( L.o_code );
        float* r = m.template arr<float>( L.o_r );
        float* a = m.template arr<float>( L.o_a );
        const __half* g = d.r_in + (size_t)m.me * L.chunk;
        const __half first = tid < n ? g[tid] : __half( 0.f );
        asm volatile( "cp.async.wait_all;" ::: "memory" );
        __syncthreads();
        for( int i = tid; i < n; i += (int)blockDim.x )
        {
            const uint16_t cc = code[i];
            const int dg = code_diag( cc );
            if( cc & kCodeBad ) atomicOr( d.err, 4u );
            const float rv = ( cc & BORA_CODE_FLUID ) ? __half2float( i == tid ? first : g[i] ) : 0.f;
            r[i] = rv;
            a[i] = ( ( cc & BORA_CODE_FLUID ) && dg > 0 ) ? ( last ? wA : wC )[dg] * rv : 0.f;
        }
    }
    m.barrier();
    // ---- down ----
    for( int t = 0; t < last; ++t )
    {
        const MidLevel& L = d.L[t];
        float* b = m.template arr<float>( L.o_b );
        m.sweep( t, L.o_a, wB, [&]( int lc, float v ) { b[lc] = v; } );  // second pre-smoothing sweep
        m.barrier();
        m.residual( t );                             // A = r - S B
        m.barrier();
        m.gather( t + 1, t + 1 == last ? wC : wA );  // coarser r and its pointwise first sweep
        m.barrier();
    }
    // ---- coarsest level: damped Jacobi from zero in CTA 0 (the first sweep, pointwise,
    // came with the gather) ----
    const MidLevel& Lc = d.L[last];
    const int zc = ( d.sweeps - 1 ) % 2 == 0 ? Lc.o_a : Lc.o_b;  // the coarsest correction's array
    if( m.me == 0 && d.sweeps > 1 )
    {
        if( Lc.n <= (int)blockDim.x ) m.template coarsest<1>( Lc, d.sweeps, wC );
        else m.template coarsest<2>( Lc, d.sweeps, wC );
    }
    m.barrier();
    // ---- up ----
    for( int t = last - 1; t >= 0; --t )
    {
        const MidLevel& L = d.L[t];
        m.inject( t, t + 1 == last ? zc : d.L[t + 1].o_a );  // A = B + Z(parent)
        m.barrier();
        float* b = m.template arr<float>( L.o_b );
        m.sweep( t, L.o_a, wB, [&]( int lc, float v ) { b[lc] = v; } );
        m.barrier();
        // the level's final correction: A, or the first level's result
        if( t > 0 )
        {
            float* a = m.template arr<float>( L.o_a );
            m.sweep( t, L.o_b, wA, [&]( int lc, float v ) { a[lc] = v; } );
            m.barrier();
        }
        else
        {
            __half* g = d.z_out + (size_t)m.me * L.chunk;
            m.sweep( t, L.o_b, wA, [&]( int lc, float v ) { g[lc] = __float2half_rn( v ); } );
        }
    }
    if( last == 0 && m.me == 0 )
    {
        const float* z = m.template arr<float>( zc );
        for( int i = tid; i < Lc.n; i += (int)blockDim.x ) d.z_out[i] = __float2half_rn( z[i] );
    }
    m.barrier();  // no CTA leaves while another may still read its shared memory
}

template <bool ONE>
__global__ void __launch_bounds__( kMidThreadsMax, 1 ) k_mg_mid( const __grid_constant__ MidDesc d )
{
    mg_mid_body<ONE>( d );
}

// Batched: one cluster per simulation taking part (all of the same size; a
// simulation's offset in the launch is a multiple of it, so a cluster is one simulation's).
template <bool ONE>
__global__ void __launch_bounds__( kMidThreadsMax, 1 ) k_mg_mid_batch( const MidDesc* __restrict__ descs,
                                                                    const __grid_constant__ BoraBatchLaunch L )
{
    unsigned bid;
    mg_mid_body<ONE>( descs[bora_batch_member( L, blockIdx.x, &bid )] );
}

// Cluster size: 16 CTAs where the device co-schedules such a cluster of this kernel with
// the largest shared memory it may ask for, else 8; 0 when neither fits (the caller then
// runs these levels itself). Queried once per device.
int mid_cluster_size()
{
    static BoraPerDevice size;  // 16, 8, or 1 for "none"
    const int v = size.get( [] {
        cudaFuncSetAttribute( k_mg_mid<false>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1 );
        cudaFuncSetAttribute( k_mg_mid<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMidSmemMax );
        cudaFuncSetAttribute( k_mg_mid_batch<false>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1 );
        cudaFuncSetAttribute( k_mg_mid_batch<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMidSmemMax );
        cudaFuncSetAttribute( k_mg_mid<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMidSmemMax );
        cudaFuncSetAttribute( k_mg_mid_batch<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMidSmemMax );
        cudaGetLastError();
        auto fits = []( int ctas ) {
            cudaLaunchConfig_t cfg{};
            cfg.gridDim = dim3( ctas );
            cfg.blockDim = dim3( kMidThreadsMax );
            cfg.dynamicSmemBytes = kMidSmemMax;
            cudaLaunchAttribute attr[1];
            attr[0].id = cudaLaunchAttributeClusterDimension;
            attr[0].val.clusterDim.x = ctas;
            attr[0].val.clusterDim.y = 1;
            attr[0].val.clusterDim.z = 1;
            cfg.attrs = attr;
            cfg.numAttrs = 1;
            int clusters = 0;
            const bool ok = cudaOccupancyMaxActiveClusters( &clusters, k_mg_mid<false>, &cfg ) == cudaSuccess && clusters > 0;
            cudaGetLastError();  // a refused query leaves no error behind
            return ok;
        };
        return fits( kMidCtasMax ) ? kMidCtasMax : ( fits( 8 ) ? 8 : 1 );
    } );
    return v > 1 ? v : 0;
}

// Shared-memory layout of the levels for `ctas` CTAs: the static block (codes, neighbour,
// parent and child references of every level) first, then the values. Returns the bytes
// per CTA.
size_t mid_layout( MidDesc& d, int ctas )
{
    size_t off = 0;
    auto take = [&]( size_t bytes ) {
        const int o = (int)off;
        off += ( bytes + 15 ) & ~(size_t)15;
        return o;
    };
    d.ctas = ctas;
    d.threads = std::clamp( ( ( ( d.L[0].n + ctas - 1 ) / ctas + 31 ) / 32 ) * 32, kMidThreadsMin, kMidThreadsMax );
    for( int t = 0; t < d.n; ++t )
    {
        MidLevel& L = d.L[t];
        L.chunk = t == d.n - 1 ? L.n : ( L.n + ctas - 1 ) / ctas;
        const size_t c = (size_t)L.chunk;
        L.o_code = take( c * 2 );
        L.o_nb = take( c * 6 * 4 );
        L.o_par = t < d.n - 1 ? take( c * 4 ) : -1;
        L.o_ch = t > 0 ? take( c * 8 * 4 ) : -1;
    }
    d.static_bytes = (int)off;
    for( int t = 0; t < d.n; ++t )
    {
        MidLevel& L = d.L[t];
        const size_t c = (size_t)L.chunk;
        L.o_r = take( c * 4 );
        L.o_a = take( ( c + 1 ) * 4 );
        L.o_b = take( ( c + 1 ) * 4 );
    }
    return off;
}

// The layout of the first level it takes (2 or 3) .. coarsest, or 0 when the hierarchy does not
// have the shape this kernel handles (ending at <= 512 cells) or does not fit the cluster's
// shared memory.
int mid_describe( const BoraGridDev& g, const BoraLevelDev* levels, int nlevels, BoraTilesDev t, int ntiles, int sweeps,
                  MidDesc& d, size_t& smem )
{
    if( ntiles <= 0 || ntiles >= ( 1 << 24 ) || sweeps < 1 || nlevels < 3 ) return 0;
    if( levels[nlevels - 1].ncells > 512 ) return 0;
    const int cluster = mid_cluster_size();
    if( cluster == 0 ) return 0;
    // from level 3, or level 2 where that is the coarsest (with level 2 in it at larger sizes, a
    // V-cycle is 2 us shorter of 36 at 152 tiles, as long at 304 and 3 us longer at 2568)
    const int first = nlevels == 3 ? 2 : 3;
    if( nlevels - first > kMidMaxLevels ) return 0;
    d = MidDesc{};
    d.n = nlevels - first;
    for( int q = 0; q < d.n; ++q )
    {
        const int l = first + q;
        const BoraLevelDev& B = levels[l];
        MidLevel& L = d.L[q];
        if( ( B.kind == 0 ) != ( l <= 3 ) ) return 0;
        L.E = B.kind == 0 ? B.E : 0;
        if( l <= 3 && ( L.E != ( l == 2 ? 2 : 1 ) || B.ncells != (size_t)ntiles * L.E * L.E * L.E ) ) return 0;
        L.n = (int)B.ncells;
        L.dx = B.dx; L.dy = B.dy; L.dz = B.dz;
        L.code = B.code;
    }
    d.nbr = t.nbr; d.tile_of = t.tile_of; d.slot_of = t.slot_of;
    d.tx = g.tx; d.ty = g.ty; d.tz = g.tz;
    d.r_in = levels[first].r;
    d.z_out = levels[first].z0;
    d.sweeps = sweeps;
    smem = 0;
    if( d.L[0].n <= kMidSingleMax && ( smem = mid_layout( d, 1 ) ) <= kMidSmemMax ) return first;
    smem = mid_layout( d, cluster );
    return smem <= kMidSmemMax ? first : 0;
}

// One launch of the V-cycle kernel: `blocks` CTAs of `threads` in clusters of `ctas`.
template <class K1, class KN, class... Args>
void mid_launch( K1 single, KN clustered, int blocks, int ctas, int threads, size_t smem, cudaStream_t st, const Args&... args )
{
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3( blocks );
    cfg.blockDim = dim3( threads );
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = ctas;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = ctas == 1 ? 1 : 2;
    if( ctas == 1 ) cudaLaunchKernelEx( &cfg, single, args... );
    else cudaLaunchKernelEx( &cfg, clustered, args... );
}

}  // namespace

size_t bora_mg_mid_image_bytes( const BoraGridDev& g, const BoraLevelDev* levels, int nlevels, BoraTilesDev t, int ntiles )
{
    MidDesc d;
    size_t smem = 0;
    if( !mid_describe( g, levels, nlevels, t, ntiles, 16, d, smem ) ) return 0;
    return (size_t)d.ctas * d.static_bytes;
}

void bora_mg_mid_setup( const BoraGridDev& g, const BoraLevelDev* levels, int nlevels, BoraTilesDev t, int ntiles,
                        void* image, cudaStream_t st )
{
    MidDesc d;
    size_t smem = 0;
    if( !image || !mid_describe( g, levels, nlevels, t, ntiles, 16, d, smem ) ) return;
    d.image = static_cast<char*>( image );
    k_mg_mid_image<<<d.ctas * kImageParts, 256, 0, st>>>( d );
}

int bora_mg_mid_vcycle( const BoraGridDev& g, const BoraLevelDev* levels, int nlevels, BoraTilesDev t, int ntiles,
                        const void* image, uint32_t* err, int sweeps, cudaStream_t st, bool launch )
{
    MidDesc d;
    size_t smem = 0;
    const int first = image ? mid_describe( g, levels, nlevels, t, ntiles, sweeps, d, smem ) : 0;
    if( !first ) return 0;
    if( !launch ) return first;
    d.image = static_cast<char*>( const_cast<void*>( image ) );
    d.err = err;
    mid_launch( k_mg_mid<true>, k_mg_mid<false>, d.ctas, d.ctas, d.threads, smem, st, d );
    return first;
}

size_t bora_mg_mid_desc_bytes() { return sizeof( MidDesc ); }

int bora_mg_mid_describe( const BoraGridDev& g, const BoraLevelDev* levels, int nlevels, BoraTilesDev t, int ntiles,
                          const void* image, uint32_t* err, int sweeps, void* desc, BoraMidShape* shape )
{
    MidDesc d;
    size_t sm = 0;
    if( !image || !mid_describe( g, levels, nlevels, t, ntiles, sweeps, d, sm ) ) return 0;
    d.image = static_cast<char*>( const_cast<void*>( image ) );
    d.err = err;
    std::memcpy( desc, &d, sizeof( d ) );
    *shape = BoraMidShape{ d.ctas, d.threads, sm };
    return 1;
}

void bora_mg_mid_launch_batch( const void* descs, const BoraBatchLaunch& L, int blocks, const BoraMidShape& shape,
                               cudaStream_t st )
{
    if( blocks <= 0 || shape.ctas <= 0 || blocks % shape.ctas ) return;
    mid_launch( k_mg_mid_batch<true>, k_mg_mid_batch<false>, blocks, shape.ctas, shape.threads, shape.smem, st,
                static_cast<const MidDesc*>( descs ), L );
}
