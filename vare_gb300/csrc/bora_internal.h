// Internal host-side declarations of the GB300 FLIP substep library (not installed).
#pragma once

#include <cstddef>
#include <cstdint>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include "flip_common.cuh"

#include <atomic>
#include <utility>
#include <vector>

// ---- per-device values computed on first use ------------------------------------------
// Launch shapes and device attributes are queried once per device ordinal. Host threads
// that drive different handles (the serving layer runs one per request) may race to fill an
// entry: each computes the same value, and the entries are atomics. Declare instances with
// static storage (zero-initialised).
class BoraPerDevice
{
public:
    template <class F>
    int get( F compute )
    {
        int dev = 0;
        if( cudaGetDevice( &dev ) != cudaSuccess || dev < 0 || dev >= kMaxDevices ) return compute();
        int v = v_[dev].load( std::memory_order_acquire );
        if( v <= 0 )
        {
            v = compute();
            v_[dev].store( v, std::memory_order_release );
        }
        return v;
    }

private:
    static constexpr int kMaxDevices = 64;
    std::atomic<int> v_[kMaxDevices];
};

// ---- programmatic dependent launch ---------------------------------------------------
// The kernels of a solver iteration form a chain in which each one reads what the one
// before wrote. They are launched with programmatic stream serialisation: a kernel may
// start while its predecessor is finishing, runs the part of its prologue that touches
// only data no kernel of the chain writes (tile tables, stencil codes, index set-up), and
// then waits for the predecessor's completion (griddepcontrol.wait) before anything else.
// Each kernel of the chain allows its successor to launch as soon as all of its own CTAs
// have started (griddepcontrol.launch_dependents), so earlier kernels are never starved.
__device__ __forceinline__ void bora_pdl_trigger() { asm volatile( "griddepcontrol.launch_dependents;" ::: "memory" ); }
__device__ __forceinline__ void bora_pdl_wait() { asm volatile( "griddepcontrol.wait;" ::: "memory" ); }

// Eight consecutive floats (an x-row of a tile, 32-byte aligned) in one 256-bit access (sm_100
// and later). A lane that owns a row would otherwise read its two halves in two 16-byte accesses
// of 32-byte stride, each of which touches every sector of the warp's rows: twice the L1 sector
// accesses (929 per tile in the PCG direction kernel). Volatile, so that no access moves across
// a dependency wait or a barrier.
__device__ __forceinline__ void bora_ld8( const float* p, float* v )
{
    asm volatile( "ld.global.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                  : "=f"( v[0] ), "=f"( v[1] ), "=f"( v[2] ), "=f"( v[3] ), "=f"( v[4] ), "=f"( v[5] ), "=f"( v[6] ), "=f"( v[7] )
                  : "l"( p ) );
}
__device__ __forceinline__ void bora_st8( float* p, const float* v )
{
    asm volatile( "st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"( p ), "f"( v[0] ), "f"( v[1] ), "f"( v[2] ),
                  "f"( v[3] ), "f"( v[4] ), "f"( v[5] ), "f"( v[6] ), "f"( v[7] )
                  : "memory" );
}

template <typename... KArgs, typename... Args>
cudaError_t bora_launch_pdl( void ( *kernel )( KArgs... ), dim3 grid, dim3 block, size_t smem, cudaStream_t st,
                             Args&&... args )
{
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx( &cfg, kernel, std::forward<Args>( args )... );
}

// ---- scan ---------------------------------------------------------------------------
size_t bora_scan_scratch_elems( size_t n );
int bora_device_scan( const uint32_t* in, uint32_t* out, size_t n, uint32_t* scratch, uint32_t* total, cudaStream_t st );

// ---- particle arrays (structure of arrays) -------------------------------------------
struct BoraParticlesDev
{
    float* px;
    float* py;
    float* pz;
    float* vx;
    float* vy;
    float* vz;
    int32_t* id;  // < 0: killed in the last step
    float* vort;  // Particles::vorticity / ::curvature (post-processing), or null while unused
    float* curv;
};

// ---- cell fields over active slots x 512 ----------------------------------------------
struct BoraCellsDev
{
    float* mass;
    float* surf;  // particle count touching the cell (PointsToCountField)
    float* pres;
    float* vx;    // grid velocity after P2G and collider velocity ("velo")
    float* vy;
    float* vz;
    float* cx;    // projected grid velocity ("comp")
    float* cy;
    float* cz;
    uint8_t* flag;
    uint16_t* code;
    float* b;
};

// Tile tables.
struct BoraTilesDev
{
    const int32_t* slot_of;   // [virtual tiles] -> slot or -1
    const int32_t* tile_of;   // [slots] -> virtual tile linear index
    const int32_t* nbr;       // [slots * 27] -> neighbour slot or -1
};

// The solver's tiles: the active tiles that hold at least one fluid cell, in slot order. The other
// active tiles (the margin the activation rule adds around the particles: a sixth of the tiles of
// the 256^3 dam break) have no unknowns, so no kernel of the solve visits them: their entries in
// the solver's vectors are neither written nor read, which also keeps more of the vectors in L2
// (256^3 plain step: 22.3 -> 18.5 ms of GPU time; mixed 4.92 -> 4.74 ms). tab: two int4
// per solver tile, (-x, +x, -y, +y) and (-z, +z, own, 0): the slots of the face neighbours (-1: not
// a solver tile) and its own.
struct BoraSolveTilesDev
{
    const int4* tab;
    const uint32_t* count;  // their number, on the device
    int n;                  // the same on the host, once known
    const int32_t* nbr;     // the active tiles' neighbour table (BoraTilesDev), for the check of the codes
};

// Scalars that the solver kernels exchange on the device (ring of FP64 reductions).
#define BORA_RING 64
// Largest grid of a kernel that reduces through BoraReduceDev::partials (one slot pair per
// block). Every such launcher clamps its grid to this, and the handle sizes the partials
// buffer for at least this many blocks.
constexpr int kBoraMaxReduceBlocks = 152 * 16;
struct BoraReduceDev
{
    double* ring;        // [BORA_RING * 4]: slot values
    double* partials;    // [max blocks * 2]
    uint32_t* done;      // [BORA_RING] block-arrival counters
    uint32_t* err;       // set non-zero by a kernel that met an inconsistent stencil code
    double* mirror;      // [BORA_RING] host-mapped copy of the slot values, or null
    // the solver chain's sums, finished by the kernel that consumes them (reduce.cuh): one
    // double-float partial per producer block, and the finished values as double-float pairs
    float2* part_dq;     // [kBoraMaxReduceBlocks] d.q, from the direction kernel
    float2* part_rz;     // r.z, from the preconditioner's last kernel
    float2* part_rr;     // r.r, from the residual update
    float2* ringf;       // [BORA_RING]
};

// ---- launchers -----------------------------------------------------------------------
void bora_launch_bin( const BoraGridDev& g, BoraParticlesDev p, size_t n, uint32_t* vkey, uint8_t* tile_flag, cudaStream_t st );
void bora_launch_activate( const BoraGridDev& g, const uint8_t* tile_flag, uint32_t* act, cudaStream_t st );
// FLIPMethod::fillWaterTank: count (write = false) or write the tank's particles.
void bora_launch_tank( const BoraGridDev& g, int hh, int per_cell, float3 tr, float3 sc, uint32_t* count,
                       const uint32_t* offset, BoraParticlesDev p, size_t base, int32_t first_id, bool write,
                       cudaStream_t st );
void bora_launch_tile_assign( const BoraGridDev& g, const uint32_t* act, const uint32_t* excl, int32_t* slot_of,
                              int32_t* tile_of, cudaStream_t st );
void bora_launch_tile_nbrs( const BoraGridDev& g, int ntiles, const int32_t* slot_of, const int32_t* tile_of,
                            int32_t* nbr, cudaStream_t st );
void bora_launch_hist( size_t n, const uint32_t* vkey, const int32_t* slot_of, uint32_t outside_key, uint32_t* key,
                       uint32_t* count, uint32_t* err, cudaStream_t st );
void bora_launch_scatter( size_t n, const uint32_t* key, const uint32_t* start, uint32_t* count, uint32_t* idx,
                          cudaStream_t st );
void bora_launch_order_bins( size_t nbins, const uint32_t* start, uint32_t* idx, cudaStream_t st );
void bora_launch_p2g( const BoraGridDev& g, int ntiles, BoraTilesDev t, BoraParticlesDev p, const uint32_t* idx,
                      const uint32_t* start, BoraCellsDev c, cudaStream_t st );
// tile_fluid: 1 for the tiles with a fluid cell
void bora_launch_rhs( const BoraGridDev& g, int ntiles, BoraTilesDev t, BoraCellsDev c, uint32_t* nfluid, uint8_t* tile_fluid,
                      cudaStream_t st );
// list[stride * q + offset] = the q-th flagged of n items (flags 0 or 1, readable up to a multiple of 16);
// their number on the device and in mapped host memory
void bora_launch_flag_list( int n, const uint8_t* flags, int32_t* list, int stride, int offset, uint32_t* count,
                            uint32_t* host_count, cudaStream_t st );
// the same flags from stencil codes that the caller has set
void bora_launch_tile_fluid( int ntiles, const uint16_t* code, uint8_t* tile_fluid, cudaStream_t st );
// the solver's tile table and count (also written to host_count, mapped host memory) from the flags
void bora_launch_solve_tiles( int ntiles, BoraTilesDev t, const uint8_t* tile_fluid, int4* tab, uint32_t* count,
                              uint32_t* host_count, cudaStream_t st );
void bora_launch_vel_update( const BoraGridDev& g, int ntiles, BoraTilesDev t, BoraCellsDev c, cudaStream_t st );
void bora_launch_g2p( const BoraGridDev& g, int ntiles, size_t nsorted, BoraTilesDev t, const uint32_t* start, BoraCellsDev c,
                      BoraParticlesDev src, const uint32_t* idx, BoraParticlesDev dst, float* adj, float dt,
                      uint32_t* nkilled, uint32_t* vkey, uint8_t* tile_flag, cudaStream_t st );
// ---- post-processing (FLIPMethod::postProcess) ------------------------------------------
void bora_launch_splat( const BoraGridDev& g, int ntiles, BoraTilesDev t, const uint32_t* start, const uint32_t* idx,
                        BoraParticlesDev p, BoraCellsDev c, cudaStream_t st );
// labels: ntiles * 512 + tiles-table entries; returns the number of kernels launched
int bora_tank_scan_launches( const BoraGridDev& g, int ntiles, BoraTilesDev t, float* surf, uint32_t* labels,
                             uint32_t* err, cudaStream_t st );
cudaError_t bora_launch_redistance( const BoraGridDev& g, int ntiles, BoraTilesDev t, const float* in, float* out,
                                    cudaStream_t st );
// curl of velo -> (wx, wy, wz); normals of surf -> comp; curvature of the normals -> pres
void bora_launch_surface_fields( const BoraGridDev& g, int ntiles, BoraTilesDev t, BoraCellsDev c, float* wx, float* wy,
                                 float* wz, cudaStream_t st );
void bora_launch_particle_attributes( const BoraGridDev& g, const int32_t* slot_of, size_t np, BoraParticlesDev p,
                                      const float* wx, const float* wy, const float* wz, const float* curvature,
                                      float3 scale, float dis, cudaStream_t st );

// ---- sparse -> VDB leaf export (FieldCast convertSurfaceVDB / convertVelocityVDB) ------
// Candidate leaves: four ints each, the voxel origin and the tile's slot or -1 (band leaf).
// bora_launch_vdb_leaves: those of the active tiles. A launch with flag != null flags the
// candidates that have an active voxel; one with keep != null writes the `n` kept ones (indices
// keep[q]) packed: origin 3 ints, mask 8 x 64 bits, val 512 (surface) or 3 x 512 (velocity) floats.
struct BoraVdbOut
{
    int n;                // leaves of this launch
    const int4* leaf;
    uint8_t* flag;
    const int32_t* keep;
    int32_t* origin;
    uint64_t* mask;
    float* val;
};
void bora_launch_vdb_leaves( const BoraGridDev& g, int ntiles, const int32_t* tile_of, int4* leaf, cudaStream_t st );
void bora_launch_vdb_surface( const BoraGridDev& g, const float* scale, const float* translate, const BoraVdbOut& o,
                              const float* surf, float bg, int tank, float level, cudaStream_t st );
void bora_launch_vdb_velocity( const BoraGridDev& g, const float* scale, const BoraVdbOut& o, const float* vx, const float* vy,
                               const float* vz, cudaStream_t st );
// three component fields <-> x, y, z interleaved (n cells, a multiple of 4)
void bora_launch_interleave( size_t n, const float* x, const float* y, const float* z, float* out, cudaStream_t st );
void bora_launch_deinterleave( size_t n, const float* in, float* x, float* y, float* z, cudaStream_t st );
int bora_vdb_level_index( float level, float min_y, float dx );
// tile coordinates (3 ints each) of the water tank's border band (FieldCast.h:398-440)
void bora_vdb_band_tiles( const BoraGridDev& g, const float* scale, const float* translate, float level,
                          std::vector<int32_t>& tiles );

void bora_launch_to_soa( size_t n, const float* pos, const float* vel, int space, const float* translate,
                         const float* scale, BoraParticlesDev p, size_t offset, int32_t first_id, cudaStream_t st );

// ---- pressure solve -------------------------------------------------------------------
struct BoraSolverDev
{
    float2* x;      // pressure iterate of the refinement as a double-float pair (hi, lo): ~48 bits
    float* e;       // inner correction
    float* r;       // residual
    float* d[2];    // search directions (ping-pong)
    float* q;       // A d
    float* z;       // preconditioned residual
    float* minv;    // squared block-MIC(0) inverse pivots, each row of a tile rotated (projection.cu)
};

// (ntiles: an upper bound for the grid; the kernels read the number of solver tiles on the device)
void bora_launch_mic_factor( int ntiles, BoraSolveTilesDev t, const uint16_t* code, float* minv, cudaStream_t st );
// r = b, x = 0, e = 0, d = 0, q = 0; partial sums of ||b||^2 and max|b| -> ring slots
void bora_launch_solve_init( int ntiles, BoraSolveTilesDev t, const float* b, BoraSolverDev s, BoraReduceDev red,
                             int slot_norm2, int slot_max, cudaStream_t st );
// r -= alpha q; z = M^-1 r; partial sums of rz and rr (alpha = rz_in / dq, or 0 when slot_rz_in < 0; dq is
// finished from the direction kernel's partials into slot_dq_in). bora_pcg_update_grid: its blocks.
int bora_pcg_update_grid( int ntiles );
void bora_launch_pcg_update( BoraSolveTilesDev t, BoraSolverDev s, BoraReduceDev red, int slot_rz_in, int slot_dq_in,
                             cudaStream_t st );
int bora_pcg_direction_grid( int ntiles );
// One refinement pass of the plain form's inner PCG in one cooperative launch with bounded
// grid barriers (projection.cu). Outputs: ring slots slot_a_rz / slot_a_dq (the last
// update's alpha, whose e += alpha d is pending), part_rr[0] (the last r.r), *iters. bar: two
// zeroed words; part: 3 * bora_pcg_persistent_grid() doubles. never_release: every barrier
// wait runs out (a test of the error path). Returns 0, or -1 when the launch is refused.
#define BORA_REDUCE_ERR_BARRIER 0x100u  // a grid barrier wait ran out
int bora_pcg_persistent_grid();
int bora_launch_pcg_persistent( BoraSolveTilesDev t, const uint16_t* code, BoraSolverDev s, BoraReduceDev red,
                                int dsel, int slot_rz_prev, int max_inner, double target, int slot_a_rz, int slot_a_dq,
                                uint32_t* iters, unsigned* bar, double* part, bool never_release, cudaStream_t st );
// The same for systems of up to 608 solver tiles, one warp per tile with its vectors in
// registers (projection.cu). ||r|| is tested every `check` iterations; `beyond` more follow one that
// reaches the target. No update is pending afterwards (e is complete); slot_a_rz: r.z before
// the last update. words: bora_pcg_resident_words_bytes() of device memory, zeroed once; the launch
// uses the tags tag .. tag + 2 max_inner, which no earlier launch over these words may have used.
int bora_pcg_resident_warps( int nft );  // warps per block, 0: too large
size_t bora_pcg_resident_words_bytes();
int bora_launch_pcg_resident( BoraSolveTilesDev t, const uint16_t* code, BoraSolverDev s, BoraReduceDev red, int dsel,
                              int slot_rz_prev, int max_inner, int check, int beyond, double target, int slot_a_rz,
                              uint32_t* iters, void* words, uint32_t tag, bool never_release, cudaStream_t st );
// d' = z + beta d; q = A d'; partial sums of dq (beta = rz_new / rz_old, or 0 when slot_rz_old < 0). Finishes rz
// and rr from nparts producer blocks' partials into slot_rz_new and slot_rr (host_rr: rr also for the host).
void bora_launch_pcg_direction( BoraSolveTilesDev t, const uint16_t* code, BoraSolverDev s, int dsel_in, BoraReduceDev red, int nparts, int slot_rz_new, int slot_rr, int slot_rz_old,
                                int slot_a_rz, int slot_a_dq, bool host_rr, cudaStream_t st );
// x = the last step's pressure on fluid cells, read through the previous tile table (the warm start)
void bora_launch_solve_warm( int ntiles, const uint16_t* code, const int32_t* tile_of, const int32_t* slot_prev,
                             const float* pres, BoraSolverDev s, cudaStream_t st );
// x += e (and the last update's pending alpha d) in double-float; e = 0; q = 0; finishes that update's rr into
// slot_rr (also for the host)
void bora_launch_refine_accumulate( BoraSolveTilesDev t, const uint16_t* code, BoraSolverDev s, int dsel, BoraReduceDev red,
                                    int nparts, int slot_rr, int slot_a_rz, int slot_a_dq, cudaStream_t st );
// r = b - A x in double-float (stored FP32); ||r||^2 and max|r| -> ring slots
void bora_launch_refine_residual( BoraSolveTilesDev t, const float* b, const uint16_t* code, BoraSolverDev s,
                                  BoraReduceDev red, int slot_norm2, int slot_max, cudaStream_t st );
// pres = (float) x on fluid cells, 0 elsewhere
void bora_launch_write_pressure( int ntiles, const uint16_t* code, const float2* x, float* pres, cudaStream_t st );


// ---- multigrid preconditioner (mixed form) ----------------------------------------------
struct BoraLevelDev
{
    int kind;          // 0 = tiled (E cells per tile edge), 1 = dense grid
    int E;             // tiled levels: 8, 4, 2, 1
    int level;         // 0 = fine grid
    int nx, ny, nz;    // cells of this level inside the domain
    int dx, dy, dz;    // dense storage extent (dense levels)
    size_t ncells;     // stored cells
    uint8_t* type;     // BORA_FLUID / BORA_AIR / BORA_SOLID / BORA_MASKED
    uint16_t* code;    // stencil code (fine-code layout)
    __half* r;         // level residual (levels >= 1), stencil units
    __half* z0;        // correction (pre-smoothed, then final)
    __half* z1;        // correction after prolongation + one sweep
};

// The tiled levels' passes of a V-cycle (mg_passes.cu): level l (E = 8, 4 or 2) pre-smoothed
// and restricted into level l + 1's r (down), or prolonged from the coarser correction ec and
// post-smoothed (up: level 0 into the PCG's z with partial sums of r.z, the others into z1).
// scratch: an FP32 vector of level 0's size. Level 0's down passes first apply the PCG's
// residual update r -= alpha q, alpha = rz / dq of slots slot_rz_in and slot_dq_in (none when
// slot_rz_in < 0; the first pass finishes dq from the direction kernel's partials), with partial
// sums of the updated r.r; slot_rr gives the scale.
int bora_mg_pass_grid( int E, int ntiles, int v );  // v < 0: level 0's fixed up-2 shape
void bora_mg_pass_down( const BoraLevelDev* levels, int l, const BoraSolveTilesDev& t, float* r0, const float* q,
                        float* scratch, const BoraReduceDev& red, int slot_rr, int slot_rz_in, int slot_dq_in,
                        cudaStream_t st );
void bora_mg_pass_up( const BoraLevelDev* levels, int l, const __half* ec, const BoraSolveTilesDev& t, const float* r0,
                      float* scratch, const BoraReduceDev& red, int slot_rr, float* z, cudaStream_t st );

// ---- launch-shape autotuner (tune.cu) ------------------------------------------------------
// Kernel groups with interchangeable launch shapes (bit-identical results): the multigrid
// passes of levels 0, 1, 2, for single simulations and for batches.
enum BoraTuneGroup
{
    kBoraTuneL0 = 0, kBoraTuneL1, kBoraTuneL2, kBoraTuneL0Batch, kBoraTuneL1Batch, kBoraTuneL2Batch, kBoraTuneGroups
};
struct BoraTunePick
{
    int variant;  // the launch shape to use
    bool timed;   // still measuring: time this launch (BoraTuneTimer)
};
int bora_tune_variants( int group );
int bora_tune_default( int group );
BoraTunePick bora_tune_pick( int group, int units );  // units: the work's size (tiles)
// Brackets the launches of a pick with events on the stream while the group is measured.
struct BoraTuneTimer
{
    bool timed;
    int group, units, variant;
    cudaStream_t st;
    cudaEvent_t a = nullptr;
    BoraTuneTimer( const BoraTunePick& p, int group, int units, cudaStream_t st );
    ~BoraTuneTimer();
    BoraTuneTimer( const BoraTuneTimer& ) = delete;
    BoraTuneTimer& operator=( const BoraTuneTimer& ) = delete;
};
// Fold the timings of completed launches into the table (call after a stream synchronize).
void bora_tune_resolve();

// Cell types and stencil codes of levels 1 .. nlevels - 1 (levels[0] = fine, given; at most 16).
// mid_image: the buffer for the coarse levels' cluster image (bora_mg_mid_image_bytes), or null.
// Returns its kernel launches.
int bora_mg_setup( const BoraGridDev& g, BoraLevelDev* levels, int nlevels, BoraTilesDev t, void* mid_image, cudaStream_t st );
// One preconditioned PCG update: r -= alpha q (alpha = rz / dq of slots slot_rz_in and slot_dq_in,
// none when slot_rz_in < 0), then one V-cycle z = M^-1 r (FP32 in and out, FP16 inside, scaled by
// 1 / sqrt(ring[slot_scale])); partial sums of r.r and r.z, bora_mg_pass_grid( 8, ntiles, -1 ) blocks each.
// Kernel launches of one bora_mg_vcycle call for this hierarchy.
int bora_mg_vcycle_launches( const BoraGridDev& g, const BoraLevelDev* levels, int nlevels, BoraTilesDev t,
                             const void* mid_image );
// Level 2 or 3 .. coarsest of a V-cycle in one thread-block cluster out of distributed shared
// memory (mg_mid.cu). bora_mg_mid_image_bytes: the device buffer its per-step static image
// needs, 0 when the hierarchy does not have the shape or size it handles;
// bora_mg_mid_setup: lay the image out (once per step, after bora_mg_setup's codes);
// bora_mg_mid_vcycle: the first level that it runs, 2 or 3 (launching the kernel when `launch`),
// 0 when the caller must run them all itself.
size_t bora_mg_mid_image_bytes( const BoraGridDev& g, const BoraLevelDev* levels, int nlevels, BoraTilesDev t, int ntiles );
void bora_mg_mid_setup( const BoraGridDev& g, const BoraLevelDev* levels, int nlevels, BoraTilesDev t, int ntiles,
                        void* image, cudaStream_t st );
int bora_mg_mid_vcycle( const BoraGridDev& g, const BoraLevelDev* levels, int nlevels, BoraTilesDev t, int ntiles,
                        const void* image, uint32_t* err, int sweeps, cudaStream_t st, bool launch );
void bora_mg_vcycle( const BoraGridDev& g, const BoraLevelDev* levels, int nlevels, BoraTilesDev t, BoraSolveTilesDev ft,
                     const void* mid_image, float* r, const float* q, float* z, float* scratch, BoraReduceDev red, int slot_rz_in,
                     int slot_dq_in, int slot_scale, int coarse_sweeps, cudaStream_t st );
// ---- batched solve: several simulations, one launch per kernel ---------------------------
// A batched launch packs the blocks of the simulations taking part back to back into one
// 1-D grid: simulation k owns blocks start[k] .. start[k+1] - 1, exactly the grid its own
// single-simulation launch of that kernel would use (grid[], fixed by its tile count alone),
// and no block when it sits the launch out. Each simulation reduces into its own ring, so
// its block indices, grid size, arithmetic and summation order are the same alone and in
// any batch, and no block of a batched launch idles. Arguments come from device arrays.
enum BoraMemberGrid
{
    kGridDir = 0, kGridCells, kGridResidual,
    kGridPass0, kGridPass0R, kGridPass1, kGridPass2,  // the multigrid passes of levels 0, 1, 2 (mg_passes.cu);
                                                      // 0R: level 0's down 1 and up 2, which reduce
    kGridCount
};
struct BoraMemberSolve
{
    int ntiles;            // active tiles (the pressure's)
    BoraSolveTilesDev ft;  // the solver's tiles
    const uint16_t* code;
    const float* b;
    float* pres;
    BoraSolverDev sv;
    BoraReduceDev red;
    BoraLevelDev L[4];     // multigrid levels 0..3 (level 3: one cell per tile)
    const __half* z3;      // level 3's correction, written by the coarse cluster kernel
    int grid[kGridCount];  // this simulation's own grid per kernel
};
struct BoraMemberSlots  // ring slots of one batched launch sequence
{
    int active;                          // 0: this simulation sits the launch out
    int dsel;                            // which search-direction buffer is the current one
    int rz_new, rr_new, rz_old, a_rz, a_dq;  // direction (finishes rz_new and rr_new; beta = rz_new / rz_old; pending
                                             // alpha); refinement: rr_new, a_rz, a_dq
    int chk;                             // the host reads rr_new
    int rz_in, dq_in;                    // residual update (alpha = rz_in / dq_in; dq_in is finished there)
    int rr;                              // V-cycle: the scale's r.r
    int n2, mx;                          // solve init / refinement residual: ||r||^2, max|r|
};
struct BoraBatchLaunch
{
    const BoraMemberSolve* ms;
    const BoraMemberSlots* sl;
    const int* start;  // n + 1 block offsets of this launch (device memory)
    int n;
};
#ifdef __CUDACC__
// The simulation owning block b of a batched launch - the last k with start[k] <= b (the
// ones before it that own no block share its offset) - and the block's index in its grid.
__device__ __forceinline__ int bora_batch_member( const BoraBatchLaunch& L, unsigned b, unsigned* bid )
{
    int lo = 0, hi = L.n;
    while( hi - lo > 1 )
    {
        const int mid = ( lo + hi ) >> 1;
        if( (unsigned)__ldg( L.start + mid ) <= b ) lo = mid;
        else hi = mid;
    }
    *bid = b - (unsigned)__ldg( L.start + lo );
    return lo;
}
#endif

// The coarse cluster kernel of a batch: a simulation's descriptor (opaque, desc_bytes each;
// 0 when its hierarchy does not fit the kernel), and one launch of `blocks` CTAs: one
// cluster of `ctas` CTAs per simulation taking part (all of the same size; threads and
// shared memory for the largest: neither they nor ctas change a value's arithmetic).
struct BoraMidShape
{
    int ctas, threads;
    size_t smem;
};
size_t bora_mg_mid_desc_bytes();
int bora_mg_mid_describe( const BoraGridDev& g, const BoraLevelDev* levels, int nlevels, BoraTilesDev t, int ntiles,
                          const void* image, uint32_t* err, int sweeps, void* desc, BoraMidShape* shape );
void bora_mg_mid_launch_batch( const void* descs, const BoraBatchLaunch& L, int blocks, const BoraMidShape& shape,
                               cudaStream_t st );
// Batched launches of the solver kernels (projection.cu, multigrid.cu) with `blocks` =
// start[n] blocks in all.
void bora_launch_solve_init_batch( const BoraBatchLaunch& L, int blocks, cudaStream_t st );
void bora_launch_pcg_direction_batch( const BoraBatchLaunch& L, int blocks, cudaStream_t st );
void bora_launch_refine_accumulate_batch( const BoraBatchLaunch& L, int blocks, cudaStream_t st );
void bora_launch_refine_residual_batch( const BoraBatchLaunch& L, int blocks, cudaStream_t st );
void bora_launch_write_pressure_batch( const BoraBatchLaunch& L, int blocks, cudaStream_t st );
// pass `pass` (0, 1 down; 2, 3 up) of multigrid level l (0, 1, 2) for the batch, launch
// shape v (level 0's up 2 has a fixed shape)
void bora_launch_mg_pass_batch( int l, int pass, int v, const BoraBatchLaunch& L, int blocks, cudaStream_t st );
// this simulation's own grid per batched kernel (what its single launches use), with the
// multigrid passes of levels 0, 1, 2 in launch shapes v[0..2]
// (of a simulation with nft solver tiles)
void bora_member_grids( int nft, int* grid, const int* v );
void bora_projection_grids( int nft, int* grid );  // the kGridDir, kGridCells and kGridResidual entries

