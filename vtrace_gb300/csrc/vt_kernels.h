// vt_kernels.h — host-callable launchers of libvtrace's CUDA kernels (internal).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "vtrace.h"

namespace vt {

struct GridView;
struct LightView;
struct Counters;

// Launch shape of the persistent tracers (picked by the autotuner).
struct TraceTuning {
    uint32_t refill_min = 16;  // refill a warp when at least this many lanes are idle (1..32)
    int blocks_per_sm = 0;     // 0: as many 256-thread blocks as fit on an SM
    uint32_t persistent = 1;   // 0: one thread per ray in 8 x 4 pixel tiles, no refill
    uint32_t wavefront = 0;    // render only: shadow rays in a second pass over a compacted queue
    uint32_t tile_shape = 0;   // render tile launch: VT_TILE_* pixels per warp
    uint32_t block_warps = 4;  // render tile launch: warps per block (1, 2, 4, 8)
    bool operator==(const TraceTuning& o) const {
        return refill_min == o.refill_min && blocks_per_sm == o.blocks_per_sm && persistent == o.persistent &&
               wavefront == o.wavefront && tile_shape == o.tile_shape && block_warps == o.block_warps;
    }
};

// Rays per warp of a launch with one thread per ray.  A launch whose rays fill only a few warps per SM
// takes as long as its longest warp: the lanes of a warp take turns in the traversal (walks and
// crossings, chains of different length), so spreading the rays over more warps shortens it until
// about thirteen warps per SM share the issue slots.  96 x 64 pixels of a 256^3 scene with shadows:
// 75.8 us with 32 rays per warp, 59.4 with 8, 53.3 with 4, 53.0 with 2; 160 x 120: 77.8, 61.4, 61.5,
// 64.1; 320 x 240: 79.9, 88.1 (16: 82.8); 4,099 rays in a 512^3 scene: 53.2, 41.0, 40.9, 34.8; 64,000:
// 63.5, 89.0 (16: 71.7).  So: rays over thirteen and a half warps per SM, to the nearest power of two.
__host__ __device__ inline uint32_t lanes_per_warp(uint64_t rays, int sm_count) {
    const uint64_t warps = (uint64_t)sm_count * 27 / 2;
    uint32_t lanes = 2;
    while (lanes < 32 && rays * 181 / 128 >= warps * (lanes * 2)) lanes *= 2;
    return lanes;
}

// Render in two passes (primary rays, then the queued shadow rays); stream-ordered scratch.
cudaError_t launch_render_wavefront(const GridView& g, const vt_camera& cam,
                                    const LightView& light, uint4* out, cudaStream_t stream);

// Persistent whole-tile render whose shadow rays are queued per warp and traced in full warps.
cudaError_t launch_render_queued(const GridView& g, const vt_camera& cam, const LightView& light,
                                 uint4* out, unsigned long long* counter, const TraceTuning& tune,
                                 int sm_count, cudaStream_t stream);
cudaError_t launch_render_persistent(const GridView& g, const vt_camera& cam,
                                     const LightView& light, uint4* out,
                                     unsigned long long* counter, const TraceTuning& tune,
                                     int sm_count, cudaStream_t stream);
cudaError_t launch_trace_rays_persistent(const GridView& g, const vt_ray* rays, uint64_t n,
                                         uint4* out, unsigned long long* counter,
                                         const TraceTuning& tune, int sm_count,
                                         cudaStream_t stream);

// `tune` selects the warp tile and block shape (nullptr: 8 x 4 pixels per warp, 4 warps).
cudaError_t launch_render(const GridView& g, const vt_camera& cam, const LightView& light,
                          uint4* out, Counters* counters, cudaStream_t stream, uint32_t row0 = 0,
                          uint32_t row1 = 0, const TraceTuning* tune = nullptr);
// Warp-time phase profile of one frame (vt_phase.cu): `totals` holds phase_profile_words() words,
// zeroed, and receives per kind and phase the warp cycles, then the passes, then the warp count.
unsigned phase_profile_words();
cudaError_t launch_render_phases(const GridView& g, const vt_camera& cam, const LightView& light,
                                 uint4* out, unsigned long long* totals, cudaStream_t stream);
cudaError_t launch_trace_rays(const GridView& g, const vt_ray* rays, uint64_t n, uint4* out,
                              Counters* counters, cudaStream_t stream);

// A box of bricks: origin and extent in brick coordinates.
struct BrickBox {
    int32_t x0, y0, z0, nx, ny, nz;
};

// Scratch of the lattice passes (vt_lattice.cu): occupancy bit rows along x, y and z, one byte per
// brick for the distance passes, and a word that is nonzero when some brick has no occupied brick
// within 14.
struct LatticeScratch {
    uint32_t* rows[3] = {nullptr, nullptr, nullptr};
    uint8_t* dist = nullptr;
    uint32_t* deep = nullptr;
};
size_t lattice_scratch_bytes(int32_t bx, int32_t by, int32_t bz);  // at most 13 per brick + padding
LatticeScratch carve_lattice_scratch(void* base, int32_t bx, int32_t by, int32_t bz);  // 16-byte aligned

// Scratch of one brick build of bx x by x bz bricks.
struct BuildScratch {
    uint64_t* words = nullptr;      // bricks * 8 occupancy words (those of occupied bricks written)
    uint32_t* occ = nullptr;        // one bit per brick: it holds an occupied voxel
    uint32_t* offsets = nullptr;    // per word of occ: occupied bricks before it in its scan block
    uint32_t* block_sums = nullptr; // occupied bricks before each scan block, then upper levels
    unsigned long long* counts = nullptr;  // occupied voxels, occupied bricks
    LatticeScratch lattice;         // in the place of `words`, which the compaction reads last
    // nullptr, or build_staging_bytes(): the voxels of each occupied brick as a 512-voxel block
    // at brick * 512, written by the words pass and copied by the compaction
    void* staged = nullptr;
};
size_t build_scratch_bytes(int32_t bx, int32_t by, int32_t bz);
size_t build_staging_bytes(uint64_t bricks, uint32_t format);
// Carves BuildScratch out of one buffer of build_scratch_bytes(bx, by, bz) bytes.
BuildScratch carve_build_scratch(void* base, int32_t bx, int32_t by, int32_t bz);

// Phase 1: occupancy words, brick flags and the occupied-voxel count; phase 2: slots.
cudaError_t launch_brick_words(const void* src, uint32_t format, const uint32_t* d_palette,
                               int32_t nx, int32_t ny, int32_t nz, const BuildScratch& s,
                               cudaStream_t stream, bool nonzero_occupancy = false);
cudaError_t launch_brick_scan(const BuildScratch& s, uint64_t bricks, cudaStream_t stream);
// Dense z-fastest input (element size 1 or 4) to x-fastest; y-planes are transposed in place of
// the x and z axes.  grid.y = ceil(nx / 32) and grid.z = ny must stay within 65535.
cudaError_t launch_transpose_xz(const void* src, void* dst, size_t elem, int32_t nx, int32_t ny,
                                int32_t nz, cudaStream_t stream);
// Phase 3: directory, compacted masks and payloads.  `counts_out` (device), or nullptr: occupied bricks,
// occupied voxels.
cudaError_t launch_brick_compact(const void* src, uint32_t format, int32_t nx, int32_t ny,
                                 int32_t nz, const BuildScratch& s, uint32_t* dir,
                                 uint64_t* masks, void* payload, cudaStream_t stream,
                                 uint64_t* counts_out = nullptr);

// Words, slots, masks, payloads, directory and palette of a grid of up to kChunkBricks bricks in one
// block.  `src` (either element order), `palette` and `counts` (occupied voxels, occupied bricks) are
// device-addressable; the lattice passes follow.
constexpr uint32_t kChunkBricks = 64;
cudaError_t launch_build_chunk(const void* src, uint32_t format, bool z_fastest, const uint32_t* palette,
                               int32_t nx, int32_t ny, int32_t nz, uint32_t* pal_out, uint32_t* dir,
                               uint64_t* masks, void* payload, unsigned long long* counts,
                               cudaStream_t stream);

// Whole passes over lattices of up to this many bricks (those built without a look at the host) settle
// distances above 14 too, at each such brick over the rows in reach: a 512 x 8 x 8 chunk with one voxel 65.6 us,
// 77.8 with the distance passes launched behind the lattice passes, 83.1 with a wait to see whether they are
// needed.  Lattices of up to 15 bricks along each axis need no distances above 14: an empty 32^3 RGBA8 chunk
// 82.0 -> 63.3 us.
constexpr uint64_t kDirectBricks = 512;
// Phase 4: octant words, long-box words and the distances below 15 of empty bricks, for every
// brick or (changed != nullptr) for the bricks a change of occupancy inside `changed` can affect.
// *s.deep tells afterwards whether a brick of those has no occupied brick within 14 in a lattice of more than
// 15 bricks along some axis: its directory entry then says 15 until launch_brick_distance settles it, but for
// whole passes over up to kDirectBricks.
cudaError_t launch_brick_lattice(uint32_t* dir, uint32_t* oct, uint32_t* lng,
                                 const LatticeScratch& s, int32_t bx, int32_t by, int32_t bz,
                                 cudaStream_t stream, const BrickBox* changed = nullptr);
// Phase 5: distances (up to 31) of the bricks whose octant word is at the cap in all octants, after
// launch_brick_lattice on the same scratch, or of every empty brick (oct == nullptr: no lattice pass
// before).
cudaError_t launch_brick_distance(uint32_t* dir, const uint32_t* oct, const LatticeScratch& s,
                                  int32_t bx, int32_t by, int32_t bz, cudaStream_t stream,
                                  const BrickBox* changed = nullptr);

}  // namespace vt
