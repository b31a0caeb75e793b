// vt_grid.cu — brick re-layout of a dense voxel grid (the ingest side of vtrace's add_texture,
// lib/memory.c:286-385): x-fastest u8 palette indices or RGBA8 texels in device memory become
// an 8^3-brick directory, 512-bit occupancy masks and dense payloads of occupied bricks only.
//
// Three passes:
//   words   one thread per (brick, z-slice): reads 8 rows of 8 voxels and builds the 64-bit occupancy
//           word; 32 consecutive bricks share one word of occupancy bits
//   scan    exclusive prefix sum of those words' bit counts = each occupied brick's slot
//   compact one warp per 32 bricks (eight in small lattices): copies the words and voxels of the
//           occupied ones into their slots; writes the directory
// In the words pass a warp's lanes are 32 consecutive bricks and a block's eight warps their eight
// z-slices, so a load instruction reads 256 contiguous bytes of a row.  With lanes running over
// the slices of four bricks it read eight pieces of 32 bytes from as many planes.
// With a staging buffer (one 512-voxel block per brick, indexed by brick), the words pass also
// writes the voxels of each occupied brick there, brick-major, while it holds them, and the
// compaction copies whole staged blocks: without it the compaction re-reads the dense grid's rows,
// whose 32-byte sectors each span four bricks along x, so a grid with few occupied bricks is read
// several times over (4.8x the payload on a 1024^3 grid with 9.5% of its bricks occupied).
#include <cuda_runtime.h>

#include "vt_device.cuh"
#include "vt_kernels.h"

namespace vt {

constexpr int kScanThreads = 1024, kScanItems = 4;
constexpr uint64_t kScanBlock = (uint64_t)kScanThreads * kScanItems;

static inline uint64_t align_up(uint64_t v, uint64_t a) { return (v + a - 1) / a * a; }

static uint64_t scan_partials(uint64_t n) {
    // block totals of every level of the scan, down to a single one
    uint64_t total = 64;
    do {
        n = (n + kScanBlock - 1) / kScanBlock;
        total += align_up(n, 64);
    } while (n > 1);
    return total;
}

// The occupancy words are not read after the compaction: the lattice passes take their space.
static uint64_t words_bytes(int32_t bx, int32_t by, int32_t bz) {
    const uint64_t words = (uint64_t)bx * by * bz * 64;
    const uint64_t lattice = lattice_scratch_bytes(bx, by, bz);
    return align_up(words > lattice ? words : lattice, 256);
}

static uint64_t occ_count(uint64_t bricks) { return (bricks + 31) / 32; }

size_t build_scratch_bytes(int32_t bx, int32_t by, int32_t bz) {
    const uint64_t n = occ_count((uint64_t)bx * by * bz);
    return (size_t)(words_bytes(bx, by, bz) + align_up(n * 4, 256) * 2 +
                    align_up(scan_partials(n) * 4, 256) + 256);
}

size_t build_staging_bytes(uint64_t bricks, uint32_t format) {
    return (size_t)align_up(bricks * 512 * (format == VT_PAYLOAD_RGBA8 ? 4 : 1), 256);
}

BuildScratch carve_build_scratch(void* base, int32_t bx, int32_t by, int32_t bz) {
    const uint64_t bricks = (uint64_t)bx * by * bz;
    char* p = (char*)base;
    BuildScratch s;
    s.words = (uint64_t*)p;
    s.lattice = carve_lattice_scratch(p, bx, by, bz);
    p += words_bytes(bx, by, bz);
    const uint64_t n = occ_count(bricks);
    s.occ = (uint32_t*)p;
    p += align_up(n * 4, 256);
    s.offsets = (uint32_t*)p;
    p += align_up(n * 4, 256);
    s.block_sums = (uint32_t*)p;
    p += align_up(scan_partials(n) * 4, 256);
    s.counts = (unsigned long long*)p;
    return s;
}

struct BrickCoord {
    int32_t bxi, byi, bzi;
};

__device__ __forceinline__ BrickCoord brick_coord(uint64_t brick, int32_t bx, int32_t by) {
    const uint32_t b = (uint32_t)brick, r = b / (uint32_t)bx;  // fewer than 2^31 bricks
    BrickCoord c;
    c.bxi = (int32_t)(b - r * (uint32_t)bx);
    c.bzi = (int32_t)(r / (uint32_t)by);
    c.byi = (int32_t)(r - (uint32_t)c.bzi * (uint32_t)by);
    return c;
}

// Occupancy bits of 8 u8 voxels packed in a u64 when "occupied" means "nonzero index": the high
// bit of each byte of ((v & 0x7F..) + 0x7F..) | v is set iff the byte is nonzero; the multiply
// gathers the eight high bits into the top byte (bit k from byte k).
__device__ __forceinline__ uint32_t nonzero_bytes(uint64_t v) {
    const uint64_t hi = (((v & 0x7F7F7F7F7F7F7F7Full) + 0x7F7F7F7F7F7F7F7Full) | v) & 0x8080808080808080ull;
    return (uint32_t)(((hi >> 7) * 0x0102040810204080ull) >> 56);
}

// Occupancy bits of one 8-voxel row: bit lx set iff voxel x0+lx is inside the grid and occupied.
template <uint32_t FMT>
__device__ __forceinline__ uint32_t row_bits(const void* src, const uint8_t* lut, size_t row_base,
                                             int32_t x0, int32_t nx, bool nz = false) {
    uint32_t bits = 0;
    if (FMT == VT_PAYLOAD_U8) {
        const uint8_t* row = (const uint8_t*)src + row_base + x0;
        if (x0 + 8 <= nx && (((uintptr_t)row) & 7u) == 0) {
            const uint2 v = __ldg((const uint2*)row);
            if (nz) return nonzero_bytes(((uint64_t)v.y << 32) | v.x);
#pragma unroll
            for (int k = 0; k < 4; ++k) bits |= (uint32_t)lut[(v.x >> (8 * k)) & 0xFFu] << k;
#pragma unroll
            for (int k = 0; k < 4; ++k) bits |= (uint32_t)lut[(v.y >> (8 * k)) & 0xFFu] << (k + 4);
        } else {
            for (int k = 0; k < 8 && x0 + k < nx; ++k) {
                const uint8_t b = __ldg(row + k);
                bits |= (uint32_t)(nz ? b != 0 : lut[b]) << k;
            }
        }
    } else {
        const uint32_t* row = (const uint32_t*)src + row_base + x0;
        if (x0 + 8 <= nx && (((uintptr_t)row) & 15u) == 0) {
            const uint4 a = __ldg((const uint4*)row), b = __ldg((const uint4*)row + 1);
            const uint32_t t[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
            for (int k = 0; k < 8; ++k) bits |= (uint32_t)((t[k] >> 24) != 0u) << k;
        } else {
            for (int k = 0; k < 8 && x0 + k < nx; ++k)
                bits |= (uint32_t)((__ldg(row + k) >> 24) != 0u) << k;
        }
    }
    return bits;
}

// Z-slice lz of brick c: 8 rows of 8 voxels, zero past the grid's edge, stored as 64 elements
// (x fastest, then y) at dst (8-byte aligned for u8, 16-byte for RGBA8).
template <uint32_t FMT>
__device__ __forceinline__ void copy_slice(const void* __restrict__ src, int32_t nx, int32_t ny,
                                           int32_t nz, const BrickCoord& c, uint32_t lz,
                                           void* __restrict__ dst) {
    const int32_t z = c.bzi * 8 + (int32_t)lz, x0 = c.bxi * 8;
    for (int ly = 0; ly < 8; ++ly) {
        const int32_t y = c.byi * 8 + ly;
        const bool row_in = z < nz && y < ny;
        const size_t row_base = (size_t)nx * ((size_t)y + (size_t)ny * (size_t)z);
        if (FMT == VT_PAYLOAD_U8) {
            const uint8_t* row = (const uint8_t*)src + row_base + x0;
            uint2 v = make_uint2(0u, 0u);
            if (row_in) {
                if (x0 + 8 <= nx && (((uintptr_t)row) & 7u) == 0) {
                    v = __ldg((const uint2*)row);
                } else {
                    uint32_t b[8] = {0, 0, 0, 0, 0, 0, 0, 0};
                    for (int k = 0; k < 8 && x0 + k < nx; ++k) b[k] = __ldg(row + k);
                    v.x = b[0] | (b[1] << 8) | (b[2] << 16) | (b[3] << 24);
                    v.y = b[4] | (b[5] << 8) | (b[6] << 16) | (b[7] << 24);
                }
            }
            ((uint2*)dst)[ly] = v;
        } else {
            const uint32_t* row = (const uint32_t*)src + row_base + x0;
            uint4 a = make_uint4(0u, 0u, 0u, 0u), b = a;
            if (row_in) {
                if (x0 + 8 <= nx && (((uintptr_t)row) & 15u) == 0) {
                    a = __ldg((const uint4*)row);
                    b = __ldg((const uint4*)row + 1);
                } else {
                    uint32_t q[8] = {0, 0, 0, 0, 0, 0, 0, 0};
                    for (int k = 0; k < 8 && x0 + k < nx; ++k) q[k] = __ldg(row + k);
                    a = make_uint4(q[0], q[1], q[2], q[3]);
                    b = make_uint4(q[4], q[5], q[6], q[7]);
                }
            }
            uint4* p = (uint4*)dst + 2 * ly;
            p[0] = a;
            p[1] = b;
        }
    }
}

// NZ: u8 grid whose palette has alpha 0 at index 0 only, so that occupancy is "index != 0" and the
// row bits come from byte arithmetic instead of palette lookups.
//
// Bound by reading the dense grid: 1 GiB of u8 voxels in and 115 MB of staged ones and words out in
// 202 us, 5.9 TB/s (0.87 of the measured copy rate); 276 us with lanes over slices, every brick's words
// written and an atomic per warp on the voxel count.
template <uint32_t FMT, bool NZ>
__global__ void __launch_bounds__(256) brick_words_kernel(const void* __restrict__ src,
                                                          const uint32_t* __restrict__ palette,
                                                          int32_t nx, int32_t ny, int32_t nz,
                                                          int32_t bx, int32_t by, uint64_t bricks,
                                                          uint64_t* __restrict__ words,
                                                          uint32_t* __restrict__ occ,
                                                          unsigned long long* occupied,
                                                          void* __restrict__ staged) {
    __shared__ uint8_t lut[256];
    __shared__ uint32_t s_any[8], s_count[8];
    if (FMT == VT_PAYLOAD_U8 && !NZ) {
        for (int i = threadIdx.x; i < 256; i += blockDim.x)
            lut[i] = (uint8_t)((__ldg(palette + i) >> 24) != 0u);
        __syncthreads();
    }
    const uint32_t lane = threadIdx.x & 31u, lz = threadIdx.x >> 5;
    const uint64_t brick = (uint64_t)blockIdx.x * 32u + lane;
    uint64_t w = 0;
    BrickCoord c = {0, 0, 0};
    bool whole = false;  // the slice's rows are in r[], 8-byte aligned and inside the grid
    uint64_t r[8];
    if (brick < bricks) {
        c = brick_coord(brick, bx, by);
        const int32_t z = c.bzi * 8 + (int32_t)lz, x0 = c.bxi * 8;
        if (z < nz) {
            const size_t plane = (size_t)nx * (size_t)ny * (size_t)z;
            const uint8_t* base = (const uint8_t*)src + plane + (size_t)nx * (size_t)(c.byi * 8) + x0;
            if (NZ && x0 + 8 <= nx && (nx & 7) == 0 && (((uintptr_t)src) & 7u) == 0 && c.byi * 8 + 8 <= ny) {
                // whole rows, 8-byte aligned: issue the eight loads before using any
                whole = true;
#pragma unroll
                for (int ly = 0; ly < 8; ++ly) r[ly] = __ldg((const unsigned long long*)(base + (size_t)nx * ly));
#pragma unroll
                for (int ly = 0; ly < 8; ++ly) w |= (uint64_t)nonzero_bytes(r[ly]) << (8 * ly);
            } else {
                for (int ly = 0; ly < 8; ++ly) {
                    const int32_t y = c.byi * 8 + ly;
                    if (y >= ny) break;
                    const size_t row_base = plane + (size_t)nx * (size_t)y;
                    w |= (uint64_t)row_bits<FMT>(src, NZ ? nullptr : lut, row_base, x0, nx, NZ) << (8 * ly);
                }
            }
        }
    }
    const uint32_t some = __ballot_sync(0xFFFFFFFFu, w != 0);
    const uint32_t count = __reduce_add_sync(0xFFFFFFFFu, (uint32_t)__popcll(w));
    if (lane == 0) {
        s_any[lz] = some;
        s_count[lz] = count;
    }
    __syncthreads();
    uint32_t any = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) any |= s_any[k];
    if (threadIdx.x == 0) {
        occ[blockIdx.x] = any;
        uint32_t total = 0;
#pragma unroll
        for (int k = 0; k < 8; ++k) total += s_count[k];
        if (total) atomicAdd(occupied, (unsigned long long)total);
    }
    if ((any >> lane) & 1u) {
        words[brick * 8 + lz] = w;
        if (staged) {  // the brick's block in the staging buffer, slice lz
            constexpr size_t E = FMT == VT_PAYLOAD_RGBA8 ? 4 : 1;
            uint8_t* dst = (uint8_t*)staged + (brick * 512 + lz * 64) * E;
            if (whole) {
                uint4* p = (uint4*)dst;
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    p[k] = make_uint4((uint32_t)r[2 * k], (uint32_t)(r[2 * k] >> 32),
                                      (uint32_t)r[2 * k + 1], (uint32_t)(r[2 * k + 1] >> 32));
            } else {
                copy_slice<FMT>(src, nx, ny, nz, c, lz, dst);  // rows just read: cache hits
            }
        }
    }
}

// Exclusive scan of up to kScanBlock items per block, of their bit counts with BITS; block totals go
// to `sums`.  `zero` (single-block launches): a word to clear.
template <bool BITS>
__global__ void __launch_bounds__(kScanThreads) scan_block_kernel(const uint32_t* __restrict__ in,
                                                                  uint32_t* __restrict__ out,
                                                                  uint64_t n,
                                                                  uint32_t* __restrict__ sums,
                                                                  uint32_t* __restrict__ zero) {
    if (zero && threadIdx.x == 0) *zero = 0u;
    __shared__ uint32_t warp_tot[kScanThreads / 32];
    const uint64_t base = (uint64_t)blockIdx.x * kScanBlock + (uint64_t)threadIdx.x * kScanItems;
    uint32_t v[kScanItems], local = 0;
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        v[k] = base + k < n ? (BITS ? (uint32_t)__popc(in[base + k]) : in[base + k]) : 0u;
        local += v[k];
    }
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    uint32_t incl = local;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, incl, off);
        if (lane >= (uint32_t)off) incl += y;
    }
    if (lane == 31) warp_tot[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        uint32_t wt = warp_tot[lane], wi = wt;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, wi, off);
            if (lane >= (uint32_t)off) wi += y;
        }
        warp_tot[lane] = wi - wt;  // exclusive prefix of warp totals
        if (lane == 31) sums[blockIdx.x] = wi;
    }
    __syncthreads();
    uint32_t run = warp_tot[warp] + incl - local;
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        if (base + k < n) out[base + k] = run;
        run += v[k];
    }
}

__global__ void scan_add_kernel(uint32_t* __restrict__ out, uint64_t n,
                                const uint32_t* __restrict__ block_offsets) {
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] += block_offsets[i / kScanBlock];
}

// In-place exclusive scan of `n` block totals; `next` holds the totals one level up, `total` takes
// the sum of them all.
static cudaError_t scan_totals(uint32_t* sums, uint64_t n, uint32_t* next, uint32_t* total,
                               cudaStream_t stream) {
    const uint64_t blocks = (n + kScanBlock - 1) / kScanBlock;
    scan_block_kernel<false><<<(unsigned)blocks, kScanThreads, 0, stream>>>(
        sums, sums, n, blocks == 1 ? total : next, nullptr);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess || blocks == 1) return e;
    e = scan_totals(next, blocks, next + align_up(blocks, 64), total, stream);
    if (e != cudaSuccess) return e;
    scan_add_kernel<<<(unsigned)((n + 255) / 256), 256, 0, stream>>>(sums, n, next);
    return cudaGetLastError();
}

// Slot of the first occupied brick of occupancy word `w`.
__device__ __forceinline__ uint32_t first_slot(const uint32_t* offsets, const uint32_t* block_sums, uint64_t w) {
    return __ldg(offsets + w) + __ldg(block_sums + w / kScanBlock);
}

cudaError_t launch_brick_scan(const BuildScratch& s, uint64_t bricks, cudaStream_t stream) {
    // the totals of the lowest level are scanned in place; the compaction adds them to its words'
    // offsets as it reads them.  counts[1] = occupied bricks: below 2^31, its low word (the words
    // pass clears both counts).
    const uint64_t n = occ_count(bricks), blocks = (n + kScanBlock - 1) / kScanBlock;
    uint32_t* total = (uint32_t*)(s.counts + 1);
    scan_block_kernel<true><<<(unsigned)blocks, kScanThreads, 0, stream>>>(
        s.occ, s.offsets, n, blocks == 1 ? total : s.block_sums, blocks == 1 ? s.block_sums : nullptr);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess && blocks > 1)
        e = scan_totals(s.block_sums, blocks, s.block_sums + align_up(blocks, 64), total, stream);
    return e;
}

cudaError_t launch_brick_words(const void* src, uint32_t format, const uint32_t* d_palette,
                               int32_t nx, int32_t ny, int32_t nz, const BuildScratch& s,
                               cudaStream_t stream, bool nonzero_occupancy) {
    const int32_t bx = (nx + 7) / 8, by = (ny + 7) / 8, bz = (nz + 7) / 8;
    const uint64_t bricks = (uint64_t)bx * by * bz;
    const unsigned blocks = (unsigned)occ_count(bricks);
    cudaError_t e = cudaMemsetAsync(s.counts, 0, 2 * sizeof(unsigned long long), stream);
    if (e != cudaSuccess) return e;
    if (format == VT_PAYLOAD_U8 && nonzero_occupancy)
        brick_words_kernel<VT_PAYLOAD_U8, true><<<blocks, 256, 0, stream>>>(
            src, d_palette, nx, ny, nz, bx, by, bricks, s.words, s.occ, s.counts, s.staged);
    else if (format == VT_PAYLOAD_U8)
        brick_words_kernel<VT_PAYLOAD_U8, false><<<blocks, 256, 0, stream>>>(
            src, d_palette, nx, ny, nz, bx, by, bricks, s.words, s.occ, s.counts, s.staged);
    else
        brick_words_kernel<VT_PAYLOAD_RGBA8, false><<<blocks, 256, 0, stream>>>(
            src, nullptr, nx, ny, nz, bx, by, bricks, s.words, s.occ, s.counts, s.staged);
    return cudaGetLastError();
}

// A warp per 32 bricks.  Bound by copying the payloads: 102 MB and their words in and out in 42 us,
// 5.9 TB/s (74 us with a thread per slice of every brick, of which nine in ten found an empty one;
// 58 us with one brick at a time per warp).
//
// Lattices of few bricks have few such warps, and a warp takes its bricks four after four: below
// kSplitGroups groups of 32 each group is split over eight warps that take four bricks each
// (vt_grid_build_u8_noalloc of 64^3 terrain 57.5 -> 40.6 us, of 256^3 67.5 -> 52.8, and 34.2 and 50.5
// with the counts written here instead of by two copies; a graph-built 64^3 grid 79.9 -> 64.7; from 2,048
// groups on, 384^3 and 512^3, the two measure the same).
constexpr uint64_t kSplitGroups = 2048;

template <uint32_t FMT, uint32_t SPLIT>
__global__ void __launch_bounds__(256) brick_compact_kernel(
    const void* __restrict__ src, int32_t nx, int32_t ny, int32_t nz, int32_t bx, int32_t by,
    uint64_t bricks, const uint64_t* __restrict__ words, const uint32_t* __restrict__ occ,
    const uint32_t* __restrict__ offsets, const uint32_t* __restrict__ block_sums,
    uint32_t* __restrict__ dir, uint64_t* __restrict__ masks, void* __restrict__ payload,
    const void* __restrict__ staged, const unsigned long long* __restrict__ counts,
    uint64_t* __restrict__ counts_out) {
    constexpr size_t E = FMT == VT_PAYLOAD_RGBA8 ? 4 : 1;
    if (counts_out && blockIdx.x == 0 && threadIdx.x < 2) counts_out[threadIdx.x] = counts[1 - threadIdx.x];
    const uint32_t lane = threadIdx.x & 31u;
    const uint64_t warp = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint64_t group = warp / SPLIT, b0 = group * 32;
    if (b0 >= bricks) return;  // whole warps
    uint32_t left = __ldg(occ + group);
    uint32_t slot = first_slot(offsets, block_sums, group);
    const uint32_t part = (uint32_t)(warp % SPLIT);
    if (part == 0u && b0 + lane < bricks)  // distance filled in by the lattice passes
        dir[b0 + lane] = (left >> lane) & 1u ? slot + __popc(left & ((1u << lane) - 1u)) : kEmptyBit;
    // four occupied bricks at a time, eight lanes each; staged blocks in pieces of 128 contiguous
    // bytes per brick and load, all of a lane's loads in flight together
    const uint32_t mine = lane >> 3, lz = lane & 7u;
    if (SPLIT != 1u) {  // the bricks of this part: four from the 4 * part-th on
        for (uint32_t k = 0; k < 4u * part; ++k) left &= left ? left - 1u : 0u;
        uint32_t rest = left;
        for (uint32_t k = 0; k < 4u; ++k) rest &= rest ? rest - 1u : 0u;
        left ^= rest;
        slot += 4u * part;
    }
    for (; left; slot += 4) {
        uint32_t at = 32;
#pragma unroll
        for (uint32_t k = 0; k < 4; ++k) {
            if (k == mine && left) at = (uint32_t)__ffs((int)left) - 1u;
            left &= left ? left - 1u : 0u;
        }
        if (at < 32) {
            const uint64_t b = b0 + at;
            const size_t to = slot + mine;
            masks[to * 8 + lz] = __ldg(words + b * 8 + lz);
            if (staged) {
                const uint4* in = (const uint4*)((const uint8_t*)staged + b * 512 * E) + lz;
                uint4* out = (uint4*)((uint8_t*)payload + to * 512 * E) + lz;
                uint4 v[4 * E];
#pragma unroll
                for (uint32_t k = 0; k < 4 * E; ++k) v[k] = __ldg(in + 8 * k);
#pragma unroll
                for (uint32_t k = 0; k < 4 * E; ++k) out[8 * k] = v[k];
                continue;
            }
            copy_slice<FMT>(src, nx, ny, nz, brick_coord(b, bx, by), lz,
                            (uint8_t*)payload + (to * 512 + lz * 64) * E);
        }
    }
}

cudaError_t launch_brick_compact(const void* src, uint32_t format, int32_t nx, int32_t ny,
                                 int32_t nz, const BuildScratch& s, uint32_t* dir,
                                 uint64_t* masks, void* payload, cudaStream_t stream, uint64_t* counts_out) {
    const int32_t bx = (nx + 7) / 8, by = (ny + 7) / 8, bz = (nz + 7) / 8;
    const uint64_t bricks = (uint64_t)bx * by * bz;
    const bool split = occ_count(bricks) < kSplitGroups;
    const unsigned blocks = (unsigned)((occ_count(bricks) * (split ? 8 : 1) + 7) / 8);
    auto* k = format == VT_PAYLOAD_U8
                  ? (split ? brick_compact_kernel<VT_PAYLOAD_U8, 8> : brick_compact_kernel<VT_PAYLOAD_U8, 1>)
                  : (split ? brick_compact_kernel<VT_PAYLOAD_RGBA8, 8> : brick_compact_kernel<VT_PAYLOAD_RGBA8, 1>);
    k<<<blocks, 256, 0, stream>>>(src, nx, ny, nz, bx, by, bricks, s.words, s.occ, s.offsets, s.block_sums, dir,
                                  masks, payload, s.staged, s.counts, counts_out);
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------------------------
// Chunk textures (up to 64 bricks: vtrace's 16^3 chunks, 32^3): words, slots, masks, payloads and
// directory in one block, a thread per row of eight voxels, from a dense array in either order that is
// read once into shared memory.  Bound by the latency of one block and of its reads (page-locked host
// memory or device memory): 7.3 us for a 16^3 RGBA8 chunk, cold (12 with a thread per slice), where the
// words, scan, count and compaction kernels took 22 and the graph also copied its input and a template.
// ---------------------------------------------------------------------------------------------
constexpr uint32_t kChunkThreads = 512;

template <uint32_t FMT>
__global__ void __launch_bounds__(kChunkThreads) build_chunk_kernel(
    const void* __restrict__ src, uint32_t z_fastest, const uint32_t* __restrict__ palette, int32_t nx,
    int32_t ny, int32_t nz, int32_t bx, int32_t by, uint32_t bricks, uint32_t* __restrict__ pal_out,
    uint32_t* __restrict__ dir, uint64_t* __restrict__ masks, void* __restrict__ payload,
    unsigned long long* __restrict__ counts) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    constexpr size_t E = FMT == VT_PAYLOAD_RGBA8 ? 4 : 1;
    __shared__ uint32_t s_alpha[8];
    __shared__ uint32_t s_any[kChunkBricks / 32];  // bricks with an occupied voxel
    __shared__ uint32_t s_count;
    __shared__ uint8_t s_bits[kChunkBricks * 64];  // occupancy of each row
    const uint32_t t = threadIdx.x, lane = t & 31u;
    const size_t bytes = (size_t)nx * ny * nz * E, vec = ((uintptr_t)src & 15u) == 0 ? bytes / 16 : 0;
    for (size_t i = t; i < vec; i += kChunkThreads)
        reinterpret_cast<uint4*>(smem_raw)[i] = reinterpret_cast<const uint4*>(src)[i];
    for (size_t i = vec * 16 + t; i < bytes; i += kChunkThreads) smem_raw[i] = ((const unsigned char*)src)[i];
    if (FMT == VT_PAYLOAD_U8 && t < 256) {
        const uint32_t c = palette[t];
        pal_out[t] = c;
        const uint32_t m = __ballot_sync(0xFFFFFFFFu, (c >> 24) != 0u);
        if (lane == 0) s_alpha[t >> 5] = m;
    }
    if (t < kChunkBricks / 32) s_any[t] = 0u;
    if (t == 0) s_count = 0u;
    __syncthreads();
    const int32_t ex = z_fastest ? nz * ny : 1, ey = z_fastest ? nz : nx, ez = z_fastest ? 1 : nx * ny;
    // row r: brick r >> 6, z-slice (r >> 3) & 7, y r & 7; voxels past the grid's edge are 0
    auto row = [&](uint32_t r, uint32_t v[8]) -> int32_t {  // number of its voxels inside the grid
        const BrickCoord c = brick_coord(r >> 6, bx, by);
        const int32_t x0 = c.bxi * 8, y = c.byi * 8 + (int32_t)(r & 7u), z = c.bzi * 8 + (int32_t)((r >> 3) & 7u);
        const int32_t n = y < ny && z < nz ? min(8, nx - x0) : 0;
        const int32_t at = ex * x0 + ey * y + ez * z;  // at most 32768 voxels
#pragma unroll
        for (int32_t k = 0; k < 8; ++k)
            v[k] = k < n ? (FMT == VT_PAYLOAD_U8 ? (uint32_t)smem_raw[at + k * ex]
                                                 : reinterpret_cast<const uint32_t*>(smem_raw)[at + k * ex])
                         : 0u;
        return n;
    };
    const uint32_t rows = bricks * 64;
    for (uint32_t r = t; r < rows; r += kChunkThreads) {  // whole warps: half a brick each
        uint32_t v[8], bits = 0;
        const int32_t n = row(r, v);
#pragma unroll
        for (int32_t k = 0; k < 8; ++k) {
            const bool o = FMT == VT_PAYLOAD_U8 ? k < n && ((s_alpha[v[k] >> 5] >> (v[k] & 31u)) & 1u) : (v[k] >> 24) != 0u;
            bits |= (uint32_t)o << k;
        }
        s_bits[r] = (uint8_t)bits;
        const uint32_t count = __reduce_add_sync(0xFFFFFFFFu, (uint32_t)__popc(bits));
        if (lane == 0 && count) {
            atomicOr(&s_any[r >> 11], 1u << ((r >> 6) & 31u));
            atomicAdd(&s_count, count);
        }
    }
    __syncthreads();
    if (t == 0) {
        uint32_t total = 0;
#pragma unroll
        for (uint32_t w = 0; w < kChunkBricks / 32; ++w) total += __popc(s_any[w]);
        counts[0] = s_count;
        counts[1] = total;
    }
    for (uint32_t r = t; r < rows; r += kChunkThreads) {
        const uint32_t k = r >> 6, in = r & 63u;
        uint32_t slot = 0;
#pragma unroll
        for (uint32_t w = 0; w < kChunkBricks / 32; ++w)
            slot += __popc(w < (k >> 5) ? s_any[w] : (w == (k >> 5) ? s_any[w] & ((1u << (k & 31u)) - 1u) : 0u));
        const bool full = (s_any[k >> 5] >> (k & 31u)) & 1u;
        if (in == 0) dir[k] = full ? slot : kEmptyBit;  // distance filled in by the lattice passes
        if (!full) continue;
        ((uint8_t*)masks)[(size_t)slot * 64 + in] = s_bits[r];
        uint32_t v[8];
        row(r, v);
        if (FMT == VT_PAYLOAD_U8) {
            ((uint2*)payload)[(size_t)slot * 64 + in] = make_uint2(v[0] | v[1] << 8 | v[2] << 16 | v[3] << 24,
                                                                   v[4] | v[5] << 8 | v[6] << 16 | v[7] << 24);
        } else {
            uint4* out = (uint4*)payload + ((size_t)slot * 64 + in) * 2;
            out[0] = make_uint4(v[0], v[1], v[2], v[3]);
            out[1] = make_uint4(v[4], v[5], v[6], v[7]);
        }
    }
}

cudaError_t launch_build_chunk(const void* src, uint32_t format, bool z_fastest, const uint32_t* palette,
                               int32_t nx, int32_t ny, int32_t nz, uint32_t* pal_out, uint32_t* dir,
                               uint64_t* masks, void* payload, unsigned long long* counts,
                               cudaStream_t stream) {
    const int32_t bx = (nx + 7) / 8, by = (ny + 7) / 8, bz = (nz + 7) / 8;
    const uint32_t bricks = (uint32_t)(bx * by * bz);
    const size_t elem = format == VT_PAYLOAD_U8 ? 1 : 4, smem = (size_t)nx * ny * nz * elem;
    const void* kernel = format == VT_PAYLOAD_U8 ? (const void*)build_chunk_kernel<VT_PAYLOAD_U8>
                                                 : (const void*)build_chunk_kernel<VT_PAYLOAD_RGBA8>;
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)(kChunkBricks * 512 * elem));
    if (e != cudaSuccess) return e;
    if (format == VT_PAYLOAD_U8)
        build_chunk_kernel<VT_PAYLOAD_U8><<<1, kChunkThreads, smem, stream>>>(
            src, z_fastest, palette, nx, ny, nz, bx, by, bricks, pal_out, dir, masks, payload, counts);
    else
        build_chunk_kernel<VT_PAYLOAD_RGBA8><<<1, kChunkThreads, smem, stream>>>(
            src, z_fastest, palette, nx, ny, nz, bx, by, bricks, pal_out, dir, masks, payload, counts);
    return cudaGetLastError();
}

}  // namespace vt

// ---------------------------------------------------------------------------------------------
// Order conversion of dense input: z-fastest (src/voxel/rawchunk.rs:292, element (x, y, z) at
// z + nz * (y + ny * x)) to the x-fastest order the brick build reads.  Each y-plane is an
// nx x nz matrix stored row-major by x; 32 x 32 tiles are staged through shared memory so that
// both the reads (along z) and the writes (along x) are contiguous per warp.
// ---------------------------------------------------------------------------------------------
namespace vt {

template <typename T>
__global__ void __launch_bounds__(256) transpose_xz_kernel(const T* __restrict__ src,
                                                           T* __restrict__ dst, int32_t nx,
                                                           int32_t ny, int32_t nz) {
    __shared__ T tile[32][33];
    const int32_t z0 = blockIdx.x * 32, x0 = blockIdx.y * 32;
    const size_t y = blockIdx.z;
    const int32_t tx = threadIdx.x & 31, ty = threadIdx.x >> 5;  // 32 x 8 threads
#pragma unroll
    for (int32_t r = ty; r < 32; r += 8) {
        const int32_t x = x0 + r, z = z0 + tx;
        if (x < nx && z < nz) tile[r][tx] = src[(size_t)z + (size_t)nz * (y + (size_t)ny * x)];
    }
    __syncthreads();
#pragma unroll
    for (int32_t r = ty; r < 32; r += 8) {
        const int32_t z = z0 + r, x = x0 + tx;
        if (x < nx && z < nz) dst[(size_t)x + (size_t)nx * (y + (size_t)ny * z)] = tile[tx][r];
    }
}

cudaError_t launch_transpose_xz(const void* src, void* dst, size_t elem, int32_t nx, int32_t ny,
                                int32_t nz, cudaStream_t stream) {
    const dim3 grid((nz + 31) / 32, (nx + 31) / 32, ny);
    if (elem == 1)
        transpose_xz_kernel<uint8_t><<<grid, 256, 0, stream>>>((const uint8_t*)src, (uint8_t*)dst,
                                                               nx, ny, nz);
    else
        transpose_xz_kernel<uint32_t><<<grid, 256, 0, stream>>>((const uint32_t*)src,
                                                                (uint32_t*)dst, nx, ny, nz);
    return cudaGetLastError();
}

}  // namespace vt
