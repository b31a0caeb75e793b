// vt_update.cu — writing a box of voxels into a resident brick grid (chunk paging).
//
// vtrace streams its world in 16^3 chunks around the camera (src/gen/pager.rs:52-78), uploading
// one new texture per frame (src/render.rs:246-261).  Here a chunk (any box, any alignment) is
// written into an existing grid instead, in place:
//
//   1. the box is uploaded (and reordered if it is z-fastest);
//   2. one thread per (affected brick, z-slice) merges the box's voxels with the brick's current
//      payload into a new occupancy word and payload slice (scratch), and flags the brick;
//   3. the host reads the flags and old directory entries of the affected bricks, keeps the slot
//      of bricks that stay occupied, frees the slots of bricks that became empty and hands out
//      slots (free list, then the high-water mark, growing the slot arrays by doubling) to bricks
//      that became occupied;
//   4. the new words and payloads are scattered into their slots and the directory entries
//      rewritten;
//   5. the octant forward distances, the long forward boxes and the Chebyshev distances are
//      recomputed for the bricks within 14 bricks of the affected ones (distances above 14, in grids
//      that have any, within 31): a change cannot reach farther.
//
// Small boxes (a 16^3 or 32^3 chunk) take steps 1 to 4 in one block: the box is read from page-locked
// memory, the slots are handed out on the device in the order the host would, and the host learns
// what happened when it waits for the whole update.
//
// The grid afterwards traverses exactly as a grid built from the updated dense array (same
// occupancy, payload, distances and octant words; only slot numbers may differ).
#include <cuda_runtime.h>

#include <string.h>

#include <algorithm>
#include <mutex>
#include <vector>

#include "vt_api_internal.h"
#include "vt_device.cuh"
#include "vt_internal.h"

namespace vt {

struct UpdateBox {
    int32_t x0, y0, z0, w, h, d;      // voxel box
    int32_t bx0, by0, bz0, kx, ky, kz;  // affected bricks
};

// One thread per (affected brick k, z-slice lz): merge and flag.  `src` is the x-fastest box.
template <typename T>
__global__ void __launch_bounds__(256) update_merge_kernel(GridView g, UpdateBox u,
                                                           const T* __restrict__ src,
                                                           uint64_t* __restrict__ words,
                                                           T* __restrict__ payload,
                                                           uint32_t* __restrict__ flags,
                                                           uint32_t* __restrict__ old_dir,
                                                           long long* __restrict__ occ_delta) {
    const uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const uint64_t K = (uint64_t)u.kx * u.ky * u.kz;
    if (t >= K * 8) return;
    const uint64_t k = t >> 3;
    const int32_t lz = (int32_t)(t & 7);
    const int32_t bxi = u.bx0 + (int32_t)(k % u.kx);
    const int32_t byi = u.by0 + (int32_t)((k / u.kx) % u.ky);
    const int32_t bzi = u.bz0 + (int32_t)(k / ((uint64_t)u.kx * u.ky));
    const size_t b = (size_t)bxi + (size_t)g.bx * ((size_t)byi + (size_t)g.by * bzi);
    const uint32_t e = g.dir[b];
    const bool was = !brick_empty(e);
    const int32_t z = bzi * 8 + lz;
    // Only cells inside the box get new occupancy: the others keep their bits, whatever value stands for a
    // cell that is not stored (an empty brick has no payload; index 0 may be opaque), and cells past the
    // grid's faces have none.
    const uint64_t old_word = was ? g.masks[(size_t)e * 8 + lz] : 0ull;
    uint64_t word = old_word;
    T* out = payload + k * 512 + lz * 64;
    for (int32_t ly = 0; ly < 8; ++ly) {
        const int32_t y = byi * 8 + ly;
        for (int32_t lx = 0; lx < 8; ++lx) {
            const int32_t x = bxi * 8 + lx;
            T v = 0;
            if (x >= u.x0 && x < u.x0 + u.w && y >= u.y0 && y < u.y0 + u.h && z >= u.z0 && z < u.z0 + u.d) {
                v = src[(size_t)(x - u.x0) + (size_t)u.w * ((size_t)(y - u.y0) + (size_t)u.h * (z - u.z0))];
                const uint32_t rgba = sizeof(T) == 1 ? g.palette[(uint32_t)v] : (uint32_t)v;
                const uint64_t bit = 1ull << (ly * 8 + lx);
                word = (rgba >> 24) ? word | bit : word & ~bit;
            } else if (was) {
                const size_t li = (size_t)lx + 8 * (ly + 8 * lz);
                if (sizeof(T) == 1)
                    v = (T)g.payload8[(size_t)e * 512 + li];
                else
                    v = (T)g.payload32[(size_t)e * 512 + li];
            }
            out[ly * 8 + lx] = v;
        }
    }
    words[k * 8 + lz] = word;
    const long long delta = (long long)__popcll(word) - (long long)__popcll(old_word);
    if (delta) atomicAdd((unsigned long long*)occ_delta, (unsigned long long)delta);
    // the brick's flag: OR of its 8 slices (lanes 8j..8j+7 of a warp hold one brick, and are
    // active together because the thread count is a multiple of 8)
    const unsigned active = __activemask();
    uint32_t f = word != 0ull;
#pragma unroll
    for (int s = 1; s < 8; s <<= 1) f |= __shfl_xor_sync(active, f, s);
    if (lz == 0) {
        flags[k] = f;
        old_dir[k] = e;
    }
}

// One thread per (affected brick, z-slice): scatter into the assigned slot, rewrite the entry.
template <typename T>
__global__ void __launch_bounds__(256) update_scatter_kernel(GridView g, UpdateBox u,
                                                             const uint64_t* __restrict__ words,
                                                             const T* __restrict__ payload,
                                                             const uint32_t* __restrict__ slots,
                                                             uint32_t* __restrict__ dir,
                                                             uint64_t* __restrict__ masks,
                                                             T* __restrict__ dst) {
    const uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const uint64_t K = (uint64_t)u.kx * u.ky * u.kz;
    if (t >= K * 8) return;
    const uint64_t k = t >> 3;
    const int32_t lz = (int32_t)(t & 7);
    const int32_t bxi = u.bx0 + (int32_t)(k % u.kx);
    const int32_t byi = u.by0 + (int32_t)((k / u.kx) % u.ky);
    const int32_t bzi = u.bz0 + (int32_t)(k / ((uint64_t)u.kx * u.ky));
    const size_t b = (size_t)bxi + (size_t)g.bx * ((size_t)byi + (size_t)g.by * bzi);
    const uint32_t slot = slots[k];
    if (lz == 0) dir[b] = slot;  // kEmptyBit | 1 for a brick left empty: distances follow
    if (brick_empty(slot)) return;
    masks[(size_t)slot * 8 + lz] = words[k * 8 + lz];
    const T* in = payload + k * 512 + lz * 64;
    T* out = dst + (size_t)slot * 512 + lz * 64;
    for (int i = 0; i < 64; ++i) out[i] = in[i];
}

// ---- small boxes: everything but the lattice passes in one block

constexpr uint32_t kSmallBricks = 128;          // affected bricks
constexpr size_t kSmallBoxBytes = 128u << 10;   // voxels of the box, in shared memory

// Exchange area in page-locked memory.
struct SmallExchange {
    // in: slots to hand out first, in the order the host's free list gives them
    uint32_t free_slots[kSmallBricks];
    // out
    uint32_t old_dir[kSmallBricks], now[kSmallBricks];
    long long occ_delta;
    uint32_t fresh, freed;
    uint32_t grow;  // nothing was written: the slot arrays are too small
    uint32_t deep;  // as LatticeScratch::deep
    uint4 box[kSmallBoxBytes / 16];
};

struct SmallUpdate {
    uint32_t nfree;       // entries of free_slots
    uint32_t slots_used;  // then new slots from here
    uint32_t slot_capacity;
    uint32_t z_fastest;
};

// A thread per row of eight voxels.  Bound by the latency of one block and of its reads over the host
// link: 7.6 us for a 16^3 u8 chunk, cold (14 us with a thread per slice).  A chunk paged into the resident
// 1024^3 grid takes 48 us in all against 110 us with an upload, the reorder, the merge, three copies back, a
// wait, the slots' upload and the scatter around the same lattice passes (the first update after a build, which
// grows the slots, 355 us).
template <typename T>
__global__ void __launch_bounds__(1024) update_small_kernel(GridView g, UpdateBox u, SmallUpdate p,
                                                            SmallExchange* __restrict__ x,
                                                            uint32_t* __restrict__ dir,
                                                            uint64_t* __restrict__ masks,
                                                            T* __restrict__ payload) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const T* box = reinterpret_cast<const T*>(smem_raw);
    __shared__ uint32_t s_alpha[8];            // palette entries that are occupied, one bit each
    __shared__ uint32_t s_fresh[4], s_freed[4];
    __shared__ uint32_t s_slot[kSmallBricks], s_free[kSmallBricks], s_old[kSmallBricks];
    __shared__ uint8_t s_bits[kSmallBricks * 64];  // occupancy of each row after the update
    __shared__ int s_delta;
    const uint32_t K = (uint32_t)(u.kx * u.ky * u.kz), t = threadIdx.x, lane = t & 31u;
    const uint32_t n16 = (uint32_t)(((size_t)u.w * u.h * u.d * sizeof(T) + 15) / 16);
    for (uint32_t i = t; i < n16; i += blockDim.x) reinterpret_cast<uint4*>(smem_raw)[i] = x->box[i];
    // brick k: (bx0 + k % kx, ...)
    auto brick_at = [&](uint32_t k, int32_t& bxi, int32_t& byi, int32_t& bzi) {
        bxi = u.bx0 + (int32_t)(k % (uint32_t)u.kx);
        byi = u.by0 + (int32_t)(k / (uint32_t)u.kx % (uint32_t)u.ky);
        bzi = u.bz0 + (int32_t)(k / (uint32_t)(u.kx * u.ky));
        return (size_t)bxi + (size_t)g.bx * ((size_t)byi + (size_t)g.by * bzi);
    };
    for (uint32_t k = t; k < K; k += blockDim.x) {
        int32_t bxi, byi, bzi;
        const uint32_t e = dir[brick_at(k, bxi, byi, bzi)];
        s_old[k] = e;
        s_slot[k] = 0u;
        x->old_dir[k] = e;
    }
    if (sizeof(T) == 1 && t < 256) {  // the block has at least 256 threads
        const uint32_t m = __ballot_sync(0xFFFFFFFFu, (g.palette[t] >> 24) != 0u);
        if (lane == 0) s_alpha[t >> 5] = m;
    }
    if (t == 0) s_delta = 0;
    __syncthreads();
    const size_t ex = p.z_fastest ? (size_t)u.d * u.h : 1, ey = p.z_fastest ? (size_t)u.d : (size_t)u.w,
                 ez = p.z_fastest ? 1 : (size_t)u.w * u.h;
    // row r: brick r >> 6, z-slice (r >> 3) & 7, y r & 7: its voxels after the update, and which of them
    // the box holds (a bit each; 0 when it does not touch the row)
    auto merged = [&](uint32_t r, T v[8]) -> uint32_t {
        int32_t bxi, byi, bzi;
        brick_at(r >> 6, bxi, byi, bzi);
        const uint32_t e = s_old[r >> 6];
        const bool was = !brick_empty(e);
        const int32_t y = byi * 8 + (int32_t)(r & 7u), z = bzi * 8 + (int32_t)((r >> 3) & 7u);
        const bool in = z >= u.z0 && z < u.z0 + u.d && y >= u.y0 && y < u.y0 + u.h;
        const T* old = payload + ((size_t)(was ? e : 0u) * 64 + (r & 63u)) * 8;
        uint32_t held = 0;
#pragma unroll
        for (int32_t lx = 0; lx < 8; ++lx) {
            const int32_t vx = bxi * 8 + lx;
            if (in && vx >= u.x0 && vx < u.x0 + u.w) {
                v[lx] = box[ex * (size_t)(vx - u.x0) + ey * (size_t)(y - u.y0) + ez * (size_t)(z - u.z0)];
                held |= 1u << lx;
            } else {
                v[lx] = was ? old[lx] : (T)0;
            }
        }
        return held;
    };
    const uint32_t rows = K * 64;
    for (uint32_t r = t; r < rows; r += blockDim.x) {  // whole warps: half a brick each
        const uint32_t e = s_old[r >> 6];
        const uint32_t before = brick_empty(e) ? 0u : (uint32_t)((const uint8_t*)masks)[(size_t)e * 64 + (r & 63u)];
        uint32_t bits = 0;
        T v[8];
        const uint32_t held = merged(r, v);
        if (held) {
#pragma unroll
            for (int32_t lx = 0; lx < 8; ++lx) {
                const bool o = sizeof(T) == 1 ? (s_alpha[(uint32_t)v[lx] >> 5] >> ((uint32_t)v[lx] & 31u)) & 1u
                                              : ((uint32_t)v[lx] >> 24) != 0u;
                bits |= (uint32_t)o << lx;
            }
        }
        bits = (bits & held) | (before & ~held);  // cells outside the box keep theirs (see update_merge_kernel)
        s_bits[r] = (uint8_t)bits;
        const uint32_t some = __ballot_sync(0xFFFFFFFFu, bits != 0u);
        const int delta = __reduce_add_sync(0xFFFFFFFFu, __popc(bits) - __popc(before));
        if (lane == 0) {
            if (some) atomicOr(&s_slot[r >> 6], 1u);
            if (delta) atomicAdd(&s_delta, delta);
        }
    }
    __syncthreads();
    // ranks of the bricks that become occupied (fresh) and empty (freed), in brick order
    const bool lists = t < ((K + 31u) & ~31u);  // whole warps
    bool fresh = false, freed = false;
    uint32_t e0 = kEmptyBit;
    if (lists) {
        if (t < K) {
            e0 = s_old[t];
            x->now[t] = s_slot[t];
        }
        const bool w0 = !brick_empty(e0), n0 = t < K && s_slot[t] != 0u;
        fresh = n0 && !w0;
        freed = w0 && !n0;
        const uint32_t mf = __ballot_sync(0xFFFFFFFFu, fresh), md = __ballot_sync(0xFFFFFFFFu, freed);
        if (lane == 0) {
            s_fresh[t >> 5] = mf;
            s_freed[t >> 5] = md;
        }
    }
    __syncthreads();
    uint32_t rank_fresh = 0, rank_freed = 0, nfresh = 0, nfreed = 0;
    for (uint32_t w = 0; w < (K + 31u) / 32u; ++w) {
        const uint32_t below = w < (t >> 5) ? 0xFFFFFFFFu : (w == (t >> 5) ? (1u << lane) - 1u : 0u);
        rank_fresh += __popc(s_fresh[w] & below);
        rank_freed += __popc(s_freed[w] & below);
        nfresh += __popc(s_fresh[w]);
        nfreed += __popc(s_freed[w]);
    }
    const uint32_t reused = min(nfresh, nfreed + p.nfree);
    const bool grow = p.slots_used + (nfresh - reused) > p.slot_capacity;
    if (t == 0) {
        x->fresh = nfresh;
        x->freed = nfreed;
        x->grow = grow ? 1u : 0u;
        x->occ_delta = s_delta;
    }
    if (grow) return;  // block-uniform; nothing of the grid is written
    uint32_t mine = kEmptyBit | 1u;  // distances follow
    if (t < K) {
        if (s_slot[t] != 0u && !fresh) mine = e0;
        // the freed slots, in brick order, go to the end of the free list, which is used from its end
        if (freed) s_free[rank_freed] = e0;
    }
    __syncthreads();
    if (t < K) {
        if (fresh) {
            const uint32_t r = rank_fresh;
            mine = r < nfreed ? s_free[nfreed - 1u - r]
                              : (r - nfreed < p.nfree ? x->free_slots[r - nfreed] : p.slots_used + (r - nfreed - p.nfree));
        }
        s_slot[t] = mine;
    }
    __syncthreads();
    for (uint32_t r = t; r < rows; r += blockDim.x) {
        const uint32_t k = r >> 6, in = r & 63u, slot = s_slot[k];
        if (in == 0) {
            int32_t bxi, byi, bzi;
            dir[brick_at(k, bxi, byi, bzi)] = slot;
        }
        if (brick_empty(slot)) continue;
        ((uint8_t*)masks)[(size_t)slot * 64 + in] = s_bits[r];
        T v[8];
        if (!merged(r, v) && !brick_empty(s_old[k])) continue;  // the row keeps its voxels in the same slot
        T* out = payload + ((size_t)slot * 64 + in) * 8;
        if (sizeof(T) == 1) {
            uint2 q;
            q.x = (uint32_t)v[0] | (uint32_t)v[1] << 8 | (uint32_t)v[2] << 16 | (uint32_t)v[3] << 24;
            q.y = (uint32_t)v[4] | (uint32_t)v[5] << 8 | (uint32_t)v[6] << 16 | (uint32_t)v[7] << 24;
            *reinterpret_cast<uint2*>(out) = q;
        } else {
            uint4* o4 = reinterpret_cast<uint4*>(out);
            o4[0] = make_uint4((uint32_t)v[0], (uint32_t)v[1], (uint32_t)v[2], (uint32_t)v[3]);
            o4[1] = make_uint4((uint32_t)v[4], (uint32_t)v[5], (uint32_t)v[6], (uint32_t)v[7]);
        }
    }
}

// Grows the slot arrays of `g` to at least `need` slots (doubling), copying the live ones.
static int32_t grow_slots(Grid& g, uint64_t need, cudaStream_t st) {
    if (need <= g.slot_capacity) return VT_OK;
    const uint64_t cap = std::max<uint64_t>(need, g.slot_capacity * 2);
    const size_t psize = g.format == VT_PAYLOAD_U8 ? 512 : 2048;
    uint64_t* m = nullptr;
    void* p = nullptr;
    if (cudaMalloc(&m, cap * 64) != cudaSuccess || cudaMalloc(&p, cap * psize) != cudaSuccess) {
        cudaFree(m);
        cudaGetLastError();
        return fail(VT_ENOMEM, "vt_grid_update: cannot grow the brick slots");
    }
    cudaError_t e = cudaMemcpyAsync(m, g.masks, g.slot_capacity * 64, cudaMemcpyDeviceToDevice, st);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(p, g.payload, g.slot_capacity * psize, cudaMemcpyDeviceToDevice, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) {
        cudaFree(m);
        cudaFree(p);
        return cuda_fail(e, "vt_grid_update: slot copy");
    }
    // slot arrays of the build's single allocation stay allocated with it: only later ones go
    g.bytes += (g.in_block(g.masks) ? cap : cap - g.slot_capacity) * (64 + psize);
    g.free_slot_arrays();
    g.masks = m;
    g.payload = p;
    state().grid_epoch.fetch_add(1);  // the grid's device view changed
    g.slot_capacity = cap;
    return VT_OK;
}

// One small update.  The caller has checked the box; its grid is not read or written elsewhere.
static int32_t update_small(Grid& g, const void* voxels, Source src, size_t elem, uint32_t order, const UpdateBox& u) {
    State& S = state();
    std::lock_guard<std::mutex> lk(S.update_mu);
    if (!S.update_pin) {
        if (cudaHostAlloc(&S.update_pin, sizeof(SmallExchange), cudaHostAllocMapped) != cudaSuccess ||
            cudaHostGetDevicePointer(&S.update_pin_dev, S.update_pin, 0) != cudaSuccess) {
            cudaGetLastError();
            cudaFreeHost(S.update_pin);
            S.update_pin = nullptr;
            return fail(VT_ENOMEM, "vt_grid_update: page-locked exchange area");
        }
    }
    SmallExchange* x = (SmallExchange*)S.update_pin;
    SmallExchange* dx = (SmallExchange*)S.update_pin_dev;
    cudaStream_t st = S.stream;
    const int32_t bx = (int32_t)g.bx, by = (int32_t)g.by, bz = (int32_t)g.bz;
    const uint32_t K = (uint32_t)(u.kx * u.ky * u.kz);
    const BrickBox changed = {u.bx0, u.by0, u.bz0, u.kx, u.ky, u.kz};
    const size_t bytes = (size_t)u.w * u.h * u.d * elem, smem = (bytes + 15) / 16 * 16;
    cudaError_t e = wait_for_source(src, st);
    if (e != cudaSuccess) return cuda_fail(e, "vt_grid_update");
    memcpy(x->box, voxels, bytes);
    const void* kernel = elem == 1 ? (const void*)update_small_kernel<uint8_t> : (const void*)update_small_kernel<uint32_t>;
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmallBoxBytes);
    void* scr = nullptr;
    if (e == cudaSuccess) e = cudaMallocAsync(&scr, lattice_scratch_bytes(bx, by, bz), st);
    if (e != cudaSuccess) return cuda_fail(e, "vt_grid_update: scratch");
    LatticeScratch ls = carve_lattice_scratch(scr, bx, by, bz);
    ls.deep = &dx->deep;
    int32_t rc = VT_OK;
    for (int attempt = 0;; ++attempt) {
        SmallUpdate p;
        p.nfree = (uint32_t)std::min<size_t>(g.free_slots.size(), K);
        for (uint32_t i = 0; i < p.nfree; ++i) x->free_slots[i] = g.free_slots[g.free_slots.size() - 1 - i];
        p.slots_used = (uint32_t)g.slots_used;
        p.slot_capacity = (uint32_t)std::min<uint64_t>(g.slot_capacity, 0x7FFFFFFFu);
        p.z_fastest = order == VT_ORDER_Z_FASTEST ? 1u : 0u;
        const unsigned threads = std::min(1024u, std::max(256u, K * 64));
        if (elem == 1)
            update_small_kernel<uint8_t><<<1, threads, smem, st>>>(g.view(), u, p, dx, g.dir, g.masks, (uint8_t*)g.payload);
        else
            update_small_kernel<uint32_t><<<1, threads, smem, st>>>(g.view(), u, p, dx, g.dir, g.masks, (uint32_t*)g.payload);
        e = cudaGetLastError();
        if (e == cudaSuccess) e = launch_brick_lattice(g.dir, g.oct, g.lng, ls, bx, by, bz, st, &changed);
        if (e == cudaSuccess && g.deep) e = launch_brick_distance(g.dir, g.oct, ls, bx, by, bz, st, &changed);
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
        if (e != cudaSuccess) { rc = cuda_fail(e, "vt_grid_update"); break; }
        if (!x->grow) break;
        if (attempt) { rc = fail(VT_ECUDA, "vt_grid_update: slots"); break; }  // not reached: grown for it
        const uint64_t reused = std::min<uint64_t>(x->fresh, x->freed + g.free_slots.size());
        if ((rc = grow_slots(g, g.slots_used + (x->fresh - reused), st))) break;
    }
    if (rc == VT_OK && !g.deep && x->deep) {
        g.deep = true;
        e = launch_brick_distance(g.dir, g.oct, ls, bx, by, bz, st, &changed);
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
        if (e != cudaSuccess) rc = cuda_fail(e, "vt_grid_update: distances");
    }
    if (rc == VT_OK) {
        // the free list as the device used it: this update's freed slots behind the others, both from
        // the end
        for (uint32_t k = 0; k < K; ++k)
            if (!(x->old_dir[k] & kEmptyBit) && !x->now[k]) g.free_slots.push_back(x->old_dir[k]);
        const uint64_t reused = std::min<uint64_t>(x->fresh, g.free_slots.size());
        g.free_slots.resize(g.free_slots.size() - reused);
        g.slots_used += x->fresh - reused;
        g.nonempty += (uint64_t)x->fresh - x->freed;  // modular: a net decrease wraps back
        g.occupied = (uint64_t)((long long)g.occupied + x->occ_delta);
    }
    cudaFreeAsync(scr, st);
    return rc;
}

}  // namespace vt

using namespace vt;

extern "C" int32_t vt_grid_update(int32_t grid, const void* voxels, uint32_t order, uint32_t x0,
                                  uint32_t y0, uint32_t z0, uint32_t w, uint32_t h, uint32_t d) {
    Grid* g = lookup_grid(grid);
    if (!g) return fail(VT_ENOTFOUND, "vt_grid_update: unknown grid");
    if (!voxels) return fail(VT_EINVAL, "vt_grid_update: null voxels");
    if (order != VT_ORDER_X_FASTEST && order != VT_ORDER_Z_FASTEST)
        return fail(VT_EINVAL, "vt_grid_update: bad order");
    if (w == 0 || h == 0 || d == 0 || (uint64_t)x0 + w > g->nx || (uint64_t)y0 + h > g->ny ||
        (uint64_t)z0 + d > g->nz)
        return fail(VT_EINVAL, "vt_grid_update: box empty or outside the grid");
    if (g->refs.load() > 0)
        return fail(VT_EBUSY, "vt_grid_update: grid is referenced by a batch or a service");
    State& s = state();
    cudaStream_t st = s.stream;
    const size_t elem = g->format == VT_PAYLOAD_U8 ? 1 : 4;
    UpdateBox u;
    u.x0 = (int32_t)x0;
    u.y0 = (int32_t)y0;
    u.z0 = (int32_t)z0;
    u.w = (int32_t)w;
    u.h = (int32_t)h;
    u.d = (int32_t)d;
    u.bx0 = u.x0 >> 3;
    u.by0 = u.y0 >> 3;
    u.bz0 = u.z0 >> 3;
    u.kx = ((u.x0 + u.w - 1) >> 3) - u.bx0 + 1;
    u.ky = ((u.y0 + u.h - 1) >> 3) - u.by0 + 1;
    u.kz = ((u.z0 + u.d - 1) >> 3) - u.bz0 + 1;
    const uint64_t K = (uint64_t)u.kx * u.ky * u.kz;
    const size_t box = (size_t)w * h * d * elem;
    if (K <= kSmallBricks && box <= kSmallBoxBytes) {
        const Source src = source_of(voxels);
        if (src != Source::kDevice) return update_small(*g, voxels, src, elem, order, u);
    }
    auto al = [](size_t v) { return (v + 255) / 256 * 256; };
    // scratch: box (x2 for reordering), words, payloads, flags, old entries, slots, delta, lattice
    // passes
    const size_t o_box = 0, o_box2 = al(box), o_words = o_box2 + (order == VT_ORDER_Z_FASTEST ? al(box) : 0);
    const size_t o_pay = o_words + al(K * 64), o_flags = o_pay + al(K * 512 * elem);
    const size_t o_old = o_flags + al(K * 4), o_slots = o_old + al(K * 4), o_delta = o_slots + al(K * 4);
    const int32_t bx = (int32_t)g->bx, by = (int32_t)g->by, bz = (int32_t)g->bz;
    const BrickBox changed = {u.bx0, u.by0, u.bz0, u.kx, u.ky, u.kz};
    const size_t o_lat = o_delta + 256, total = o_lat + lattice_scratch_bytes(bx, by, bz);
    char* scr = nullptr;
    cudaError_t e = cudaMallocAsync((void**)&scr, total, st);
    if (e != cudaSuccess) return cuda_fail(e, "vt_grid_update: scratch");
    int32_t rc = VT_OK;
    std::vector<uint32_t> flags(K), old(K), slots(K);
    long long delta = 0;
    do {
        // 1. upload, reorder
        e = cudaMemcpyAsync(scr + o_box, voxels, box, cudaMemcpyHostToDevice, st);
        const void* src = scr + o_box;
        if (e == cudaSuccess && order == VT_ORDER_Z_FASTEST) {
            e = launch_transpose_xz(scr + o_box, scr + o_box2, elem, u.w, u.h, u.d, st);
            src = scr + o_box2;
        }
        if (e == cudaSuccess) e = cudaMemsetAsync(scr + o_delta, 0, 8, st);
        if (e != cudaSuccess) { rc = cuda_fail(e, "vt_grid_update: upload"); break; }
        // 2. merge
        const GridView v = g->view();
        const unsigned blocks = (unsigned)((K * 8 + 255) / 256);
        if (elem == 1)
            update_merge_kernel<uint8_t><<<blocks, 256, 0, st>>>(
                v, u, (const uint8_t*)src, (uint64_t*)(scr + o_words), (uint8_t*)(scr + o_pay),
                (uint32_t*)(scr + o_flags), (uint32_t*)(scr + o_old), (long long*)(scr + o_delta));
        else
            update_merge_kernel<uint32_t><<<blocks, 256, 0, st>>>(
                v, u, (const uint32_t*)src, (uint64_t*)(scr + o_words), (uint32_t*)(scr + o_pay),
                (uint32_t*)(scr + o_flags), (uint32_t*)(scr + o_old), (long long*)(scr + o_delta));
        e = cudaGetLastError();
        if (e == cudaSuccess) e = cudaMemcpyAsync(flags.data(), scr + o_flags, K * 4, cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess) e = cudaMemcpyAsync(old.data(), scr + o_old, K * 4, cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess) e = cudaMemcpyAsync(&delta, scr + o_delta, 8, cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
        if (e != cudaSuccess) { rc = cuda_fail(e, "vt_grid_update: merge"); break; }
        // 3. slots: free first, so that freed slots are reused by this update's new bricks
        uint64_t fresh = 0;
        for (uint64_t k = 0; k < K; ++k) {
            const bool was = !(old[k] & kEmptyBit), now = flags[k] != 0;
            if (was && !now) g->free_slots.push_back(old[k]);
            if (!was && now) ++fresh;
        }
        const uint64_t reuse = std::min<uint64_t>(fresh, g->free_slots.size());
        if ((rc = grow_slots(*g, g->slots_used + (fresh - reuse), st))) break;
        for (uint64_t k = 0; k < K; ++k) {
            const bool was = !(old[k] & kEmptyBit), now = flags[k] != 0;
            if (!now) {
                slots[k] = kEmptyBit | 1u;
            } else if (was) {
                slots[k] = old[k];
            } else if (!g->free_slots.empty()) {
                slots[k] = g->free_slots.back();
                g->free_slots.pop_back();
            } else {
                slots[k] = (uint32_t)g->slots_used++;
            }
        }
        // 4. scatter
        e = cudaMemcpyAsync(scr + o_slots, slots.data(), K * 4, cudaMemcpyHostToDevice, st);
        if (e != cudaSuccess) { rc = cuda_fail(e, "vt_grid_update: slots"); break; }
        const GridView v2 = g->view();
        if (elem == 1)
            update_scatter_kernel<uint8_t><<<blocks, 256, 0, st>>>(
                v2, u, (const uint64_t*)(scr + o_words), (const uint8_t*)(scr + o_pay),
                (const uint32_t*)(scr + o_slots), g->dir, g->masks, (uint8_t*)g->payload);
        else
            update_scatter_kernel<uint32_t><<<blocks, 256, 0, st>>>(
                v2, u, (const uint64_t*)(scr + o_words), (const uint32_t*)(scr + o_pay),
                (const uint32_t*)(scr + o_slots), g->dir, g->masks, (uint32_t*)g->payload);
        e = cudaGetLastError();
        // 5. octant words, long boxes and distances around the change; the distance passes only in
        // grids that have, or now get, bricks far from all occupied ones
        const LatticeScratch ls = carve_lattice_scratch(scr + o_lat, bx, by, bz);
        uint32_t deep = 0;
        if (e == cudaSuccess) e = launch_brick_lattice(g->dir, g->oct, g->lng, ls, bx, by, bz, st, &changed);
        if (e == cudaSuccess && g->deep) e = launch_brick_distance(g->dir, g->oct, ls, bx, by, bz, st, &changed);
        if (e == cudaSuccess && !g->deep) e = cudaMemcpyAsync(&deep, ls.deep, 4, cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
        if (e == cudaSuccess && deep) {
            g->deep = true;
            e = launch_brick_distance(g->dir, g->oct, ls, bx, by, bz, st, &changed);
            if (e == cudaSuccess) e = cudaStreamSynchronize(st);
        }
        if (e != cudaSuccess) { rc = cuda_fail(e, "vt_grid_update: scatter"); break; }
        uint64_t nonempty = 0;
        for (uint64_t k = 0; k < K; ++k) {
            const bool was = !(old[k] & kEmptyBit), now = flags[k] != 0;
            nonempty += (uint64_t)now - (uint64_t)was;
        }
        g->nonempty += nonempty;  // modular: a net decrease wraps back
        g->occupied = (uint64_t)((long long)g->occupied + delta);
    } while (0);
    cudaFreeAsync(scr, st);
    cudaStreamSynchronize(st);
    return rc;
}
