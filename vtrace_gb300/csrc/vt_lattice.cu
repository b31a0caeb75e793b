// vt_lattice.cu — empty-space tables of a brick grid: forward cubes, long boxes and distances.
//
// Per brick and ray octant o = (dx<0) | (dy<0)<<1 | (dz<0)<<2 (cells beyond the lattice are empty):
//   K   the largest K <= 15 such that the K x K x K bricks from it toward o are empty (octant words)
//   L_a the largest L <= 15 such that the box L bricks long along axis a and K x K across, toward
//       o, is empty (long-box words)
//   D   the Chebyshev distance to the nearest occupied brick, at most 31 (directory entries)
//
// All three come from one bit per brick.  The lattice's occupancy is kept as bit rows along each of
// the three axes (256 KB each for 128^3 bricks).  For an axis a, OR together the rows of the k x k
// cross-section from a row toward one of the four lateral sign pairs q: the run of zero bits from
// position p of that merged row M(k, q) toward +-a is the length of the empty k x k box from p.  So
//   K >= k   iff that run (a = x) is at least k: one shift-and-AND erosion tests 32 bricks at once
//   L_a       = the run in M(K, q) from the brick, at most 15: one shift and one find-first-set
// and the centred cube of radius r < 15 is the union of the eight octants' cubes of side r + 1, so
//   D         = the smallest K of the eight octants when that is below 15
// Bricks whose eight octants all reach the cap (empty in all directions for 15 bricks) are left to
// the separable distance passes at the end of this file, which the host launches when there are any; in
// lattices of few bricks the x pass looks at all rows for them.
//
// A block takes 32 bricks along the axis x 8 x 8 rows.  It reads the 36 x 36 rows within reach as
// 62-bit windows, builds the ORs of 2^p x 2^p rows (p = 0..3) in shared memory, from which M(k, q)
// is four look-ups (overlapping power-of-two blocks), and then works without barriers: one thread
// per (row, q) over k = 1, 2, ..., then one lane per brick.  Bound by instruction issue and the
// shared-memory look-ups (72 % of their rate in the y and z passes): the tables' 20 bytes per brick
// are the only global traffic of size.
//
// 128^3 bricks (1024^3 voxels, 9.5 % of the bricks occupied): rows 8 us, x 31 us, y and z 51 us,
// together 90 us where per-brick walks (distances, octants) and a pyramid of run minima (long
// boxes) took 615 us; after a 16^3 chunk's update 28 us where they took 110 us.
#include <cuda_runtime.h>

#include <algorithm>

#include "vt_device.cuh"
#include "vt_kernels.h"

namespace vt {

constexpr int32_t kCap = 15;          // K and L caps (nibbles)
constexpr int32_t kHalo = kCap - 1;   // bricks a forward box reaches past its first one
constexpr int32_t kTile = 8;          // rows per block along each lateral axis
constexpr int32_t kSpan = kTile + 2 * kHalo;  // 36 rows in reach along each
constexpr int32_t kPitch = 40;        // u64 per table line: 8-row groups of a warp in distinct banks
constexpr int32_t kRows = kTile * kTile;
constexpr int32_t kLatticeThreads = 256;  // one thread per (row, lateral sign pair)

// ORs of 2^p x 2^p rows: table p has (36 - 2^p + 1) lines.
__host__ __device__ constexpr int32_t table_lines(int p) { return kSpan - (1 << p) + 1; }
__host__ __device__ constexpr int32_t table_base(int p) {
    return p == 0 ? 0 : table_base(p - 1) + table_lines(p - 1) * kPitch;
}
constexpr int32_t kTableWords = table_base(4);       // u64
constexpr int32_t kLevelPitch = 4 * kRows + 1;       // merged rows of one k: [q][row], padded
constexpr size_t kLatticeShared = (size_t)(kTableWords + kCap * kLevelPitch) * 8;  // 73,400 B: 3 blocks per SM

__device__ __forceinline__ int32_t row_words(int32_t n) { return (n + 31) >> 5; }

// Transpose of a 32 x 32 bit matrix held one row per lane (bit i = column i).
__device__ __forceinline__ uint32_t transpose32(uint32_t x) {
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t m = 0x0000FFFFu;
#pragma unroll
    for (int s = 16; s; s >>= 1) {
        const uint32_t y = __shfl_xor_sync(0xFFFFFFFFu, x, s);
        x = (lane & s) ? ((x & ~m) | ((y >> s) & m)) : ((x & m) | ((y << s) & ~m));
        m ^= m << (s >> 1);
    }
    return x;
}

// Occupancy rows along x, y and z of the bricks of `box` (origin and extent multiples of 32 or the
// lattice's end).  A warp reads 32 x 32 bricks of the (x, y) or (x, z) plane, one ballot per line,
// and transposes the 32 words for the other axis.
__global__ void __launch_bounds__(256) lattice_rows_kernel(const uint32_t* __restrict__ dir,
                                                           LatticeScratch s, int32_t bx, int32_t by,
                                                           int32_t bz, BrickBox box) {
    if (blockIdx.x == 0 && threadIdx.x == 0) *s.deep = 0u;
    const int32_t lane = (int32_t)(threadIdx.x & 31u);
    const uint64_t t = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint64_t nwx = (uint64_t)row_words(box.nx), nwy = (uint64_t)row_words(box.ny),
                   nwz = (uint64_t)row_words(box.nz);
    const uint64_t nxy = nwx * nwy * (uint64_t)box.nz, nxz = nwx * (uint64_t)box.ny * nwz;
    if (t >= nxy + nxz) return;
    const bool plane_xy = t < nxy;
    const uint64_t i = plane_xy ? t : t - nxy;
    const int32_t x0 = box.x0 + 32 * (int32_t)(i % nwx);
    const uint64_t r = i / nwx;
    int32_t y0, z0;
    if (plane_xy) {
        y0 = box.y0 + 32 * (int32_t)(r % nwy);
        z0 = box.z0 + (int32_t)(r / nwy);
    } else {
        y0 = box.y0 + (int32_t)(r % (uint64_t)box.ny);
        z0 = box.z0 + 32 * (int32_t)(r / (uint64_t)box.ny);
    }
    const int32_t n = plane_xy ? min(32, by - y0) : min(32, bz - z0);
    const uint64_t step = plane_xy ? (uint64_t)bx : (uint64_t)bx * by;
    const uint32_t* d = dir + (uint64_t)x0 + (uint64_t)bx * ((uint64_t)y0 + (uint64_t)by * (uint64_t)z0) + lane;
    const bool in_x = x0 + lane < bx;
    uint32_t line = 0;
#pragma unroll
    for (int32_t h = 0; h < 32; h += 16) {  // sixteen loads in flight
        uint32_t e[16];
#pragma unroll
        for (int32_t j = 0; j < 16; ++j)
            e[j] = in_x && h + j < n ? __ldg(d + step * (uint64_t)(h + j)) : kEmptyBit;
#pragma unroll
        for (int32_t j = 0; j < 16; ++j) {
            const uint32_t w = __ballot_sync(0xFFFFFFFFu, !brick_empty(e[j]));
            if (lane == h + j) line = w;
        }
    }
    const uint32_t across = transpose32(line);
    const int32_t wx = row_words(bx), wy = row_words(by), wz = row_words(bz);
    if (plane_xy) {
        if (lane < n) s.rows[0][((uint64_t)z0 * by + (uint64_t)(y0 + lane)) * wx + (x0 >> 5)] = line;
        if (in_x) s.rows[1][((uint64_t)z0 * bx + (uint64_t)(x0 + lane)) * wy + (y0 >> 5)] = across;
    } else if (in_x) {
        s.rows[2][((uint64_t)y0 * bx + (uint64_t)(x0 + lane)) * wz + (z0 >> 5)] = across;
    }
}

// A block's tile: axis a, first brick along it (a0) and of its rows (t1, t2: lateral axes in
// ascending order), and the lattice's extent along them.
struct Tile {
    int32_t a0, t1, t2;
    int32_t na, n1, n2;
};

// Tile `i` of window `w` for axis A.
template <int A>
__device__ __forceinline__ Tile lattice_tile(const BrickBox& w, uint32_t i, int32_t bx, int32_t by,
                                             int32_t bz) {
    Tile t;
    const int32_t wa = A == 0 ? w.nx : (A == 1 ? w.ny : w.nz);
    const int32_t w1 = A == 0 ? w.ny : w.nx;
    const uint32_t ca = (uint32_t)(wa + 31) / 32u, c1 = (uint32_t)(w1 + kTile - 1) / kTile;
    t.a0 = (A == 0 ? w.x0 : (A == 1 ? w.y0 : w.z0)) + 32 * (int32_t)(i % ca);
    t.t1 = (A == 0 ? w.y0 : w.x0) + kTile * (int32_t)((i / ca) % c1);
    t.t2 = (A == 2 ? w.y0 : w.z0) + kTile * (int32_t)(i / ca / c1);
    t.na = A == 0 ? bx : (A == 1 ? by : bz);
    t.n1 = A == 0 ? by : bx;
    t.n2 = A == 2 ? by : bz;
    return t;
}

// The tile's rows in reach as windows of 62 bits (bit 15 + i: brick a0 + i), then the ORs of
// 2^p x 2^p of them.
__device__ __forceinline__ void lattice_tables(const uint32_t* __restrict__ rows, const Tile& t,
                                               uint64_t* tab) {
    const int32_t wn = row_words(t.na), start = t.a0 - kCap;
    const int32_t w0 = start >> 5, sh = start & 31;  // floor division: start may be negative
    for (int32_t k = threadIdx.x; k < kSpan * kSpan; k += kLatticeThreads) {
        const int32_t i2 = k / kSpan, i1 = k - i2 * kSpan;
        const int32_t c1 = t.t1 + i1 - kHalo, c2 = t.t2 + i2 - kHalo;
        uint64_t v = 0;
        if (c1 >= 0 && c1 < t.n1 && c2 >= 0 && c2 < t.n2) {
            const uint32_t* row = rows + ((uint64_t)c2 * t.n1 + (uint64_t)c1) * wn;
            const uint64_t a = w0 >= 0 && w0 < wn ? __ldg(row + w0) : 0u;
            const uint64_t b = w0 + 1 >= 0 && w0 + 1 < wn ? __ldg(row + w0 + 1) : 0u;
            const uint64_t c = w0 + 2 < wn ? __ldg(row + w0 + 2) : 0u;
            v = (a | (b << 32)) >> sh;
            if (sh) v |= c << (64 - sh);
        }
        tab[i2 * kPitch + i1] = v;
    }
    __syncthreads();
#pragma unroll
    for (int p = 1; p < 4; ++p) {
        const int32_t n = table_lines(p), h = 1 << (p - 1);
        const uint64_t* in = tab + table_base(p - 1);
        uint64_t* out = tab + table_base(p);
        for (int32_t k = threadIdx.x; k < n * n; k += kLatticeThreads) {
            const int32_t i2 = k / n, i1 = k - i2 * n;
            const uint64_t* q = in + i2 * kPitch + i1;
            out[i2 * kPitch + i1] = q[0] | q[h] | q[h * kPitch] | q[h * kPitch + h];
        }
        __syncthreads();
    }
}

// M(k, q) of a thread's row: `at` is the row's place in table 0, n1 / n2 are -1 where the lateral
// direction is negative, else 0 (the cross-section then starts k - 1 rows before it).
__device__ __forceinline__ uint64_t merged_row(const uint64_t* tab, int32_t at, int32_t n1,
                                               int32_t n2, int32_t k) {
    const int32_t p = 31 - __clz(k), off = k - (1 << p);  // compile-time: k is an unrolled index
    const uint64_t* q = tab + table_base(p) + at + (n2 * kPitch + n1) * (k - 1);
    uint64_t m = q[0];
    if (off) m |= q[off] | q[off * kPitch] | q[off * kPitch + off];
    return m;
}

// Empty run from lane `lane`'s brick (bit 15 + lane) toward +a / -a, at most 15.
__device__ __forceinline__ uint32_t run_forward(uint64_t m, uint32_t lane) {
    return (uint32_t)__ffs((int)((uint32_t)(m >> (15u + lane)) | 0x8000u)) - 1u;
}
__device__ __forceinline__ uint32_t run_backward(uint64_t m, uint32_t lane) {
    return (uint32_t)__clz((int)((uint32_t)((m << (48u - lane)) >> 32) | 0x10000u));
}

// Distance along x from brick x to the nearest occupied brick of its row, at most `cap` (<= 31).
__device__ __forceinline__ int32_t row_distance(const uint32_t* __restrict__ row, int32_t rw,
                                                int32_t x, int32_t cap) {
    const int32_t w = x >> 5, b = x & 31;
    const uint64_t mid = __ldg(row + w);
    const uint64_t up = (mid | (w + 1 < rw ? (uint64_t)__ldg(row + w + 1) << 32 : 0ull)) >> b;
    const uint64_t down = ((mid << 32) | (w > 0 ? (uint64_t)__ldg(row + w - 1) : 0ull)) << (31 - b);
    const int32_t f = up ? __ffsll((long long)up) - 1 : cap;      // bit k: brick x + k
    const int32_t g = down ? __clzll((long long)down) : cap;      // bit 63 - k: brick x - k
    return min(cap, min(f, g));
}

// Distance of a brick over the rows in reach of a lattice of few bricks; four rows' loads in flight.
__device__ __forceinline__ uint32_t direct_distance(const uint32_t* __restrict__ rows, int32_t x, int32_t y,
                                                    int32_t z, int32_t by, int32_t bz, int32_t rw) {
    constexpr int32_t R = (int32_t)kMaxBrickDistance;
    int32_t best = R;
    const int32_t y0 = max(y - R + 1, 0), y1 = min(y + R, by);
    for (int32_t k = max(z - R + 1, 0); k < min(z + R, bz); ++k)
#pragma unroll 4
        for (int32_t j = y0; j < y1; ++j) {
            const int32_t d = row_distance(rows + (uint64_t)(k * by + j) * rw, rw, x, R);
            best = min(best, max(max(abs(j - y), abs(k - z)), d));
        }
    return (uint32_t)best;
}

// What the x pass does with the distance of a brick whose octants all reach the cap.
enum class FarBricks {
    kLater,  // 15: the distance passes settle it
    kNone,   // 31: the lattice has at most 15 bricks along each axis, so those 14 around are all of it
    kHere,   // looks at all rows
};

// Axis x: octant words, distances of empty bricks, and the long-box words along x.
template <FarBricks FAR>
__global__ void __launch_bounds__(kLatticeThreads) lattice_x_kernel(
    LatticeScratch s, uint32_t* __restrict__ dir, uint32_t* __restrict__ oct,
    uint32_t* __restrict__ lng, int32_t bx, int32_t by, int32_t bz, BrickBox w) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    uint64_t* tab = reinterpret_cast<uint64_t*>(smem_raw);
    uint64_t* lev = tab + kTableWords;
    const Tile t = lattice_tile<0>(w, blockIdx.x, bx, by, bz);
    lattice_tables(s.rows[0], t, tab);
    const int32_t row = threadIdx.x & (kRows - 1), q = threadIdx.x / kRows;
    const int32_t at = ((row / kTile) + kHalo) * kPitch + (row % kTile) + kHalo;
    const int32_t n1 = (q & 1) ? -1 : 0, n2 = (q & 2) ? -1 : 0;
    // Bit-sliced K of the row's 32 bricks: the sets "K >= k" are nested, so bit j of K is the XOR of
    // the sets at the multiples of 2^j.  Forward boxes of the -x octants end where those of the
    // +x octants start, so one erosion serves both.
    uint32_t kf[4] = {0, 0, 0, 0}, kb[4] = {0, 0, 0, 0};
#pragma unroll
    for (int k = 1; k <= kCap; ++k) {
        const uint64_t m = merged_row(tab, at, n1, n2, k);
        lev[(k - 1) * kLevelPitch + q * kRows + row] = m;
        uint64_t f = ~m;
        if (k >= 2) f &= f >> 1;
        if (k >= 4) f &= f >> 2;
        if (k >= 8) f &= f >> 4;
        const int p = k >= 8 ? 8 : (k >= 4 ? 4 : (k >= 2 ? 2 : 1));
        if (k > p) f &= f >> (k - p);  // bit j: bricks j .. j + k - 1 of the merged row are empty
        const uint32_t ef = (uint32_t)(f >> kCap), eb = (uint32_t)(f >> (kCap + 1 - k));
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (k % (1 << j) == 0) {
                kf[j] ^= ef;
                kb[j] ^= eb;
            }
        if (!__any_sync(0xFFFFFFFFu, (ef | eb) != 0u)) break;  // no larger cube in these rows
    }
    __syncthreads();  // the tables are read: their space takes the K bits
    uint32_t* bits = reinterpret_cast<uint32_t*>(tab);  // [row][33]: word 4 * octant + bit
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        bits[row * 33 + 8 * q + j] = kf[j];      // octant 2 q
        bits[row * 33 + 8 * q + 4 + j] = kb[j];  // octant 2 q + 1
    }
    __syncthreads();
    const uint32_t lane = threadIdx.x & 31u;
    const int32_t x = t.a0 + (int32_t)lane;
    bool far = false;
#pragma unroll 2
    for (int32_t r = (int32_t)(threadIdx.x >> 5); r < kRows; r += kLatticeThreads / 32) {
        const int32_t y = t.t1 + r % kTile, z = t.t2 + r / kTile;
        if (y >= w.y0 + w.ny || z >= w.z0 + w.nz) continue;  // warp-uniform
        const uint32_t ow = transpose32(bits[r * 33 + lane]);
        uint32_t least = kCap, lw = 0;
#pragma unroll
        for (int o = 0; o < 8; ++o) {
            const uint32_t K = (ow >> (4 * o)) & 15u;
            least = min(least, K);
            const uint64_t m = lev[(max(K, 1u) - 1u) * kLevelPitch + (o >> 1) * kRows + r];
            lw |= ((o & 1) ? run_backward(m, lane) : run_forward(m, lane)) << (4 * o);
        }
        if (x < w.x0 + w.nx) {
            const uint64_t b = (uint64_t)x + (uint64_t)bx * ((uint64_t)y + (uint64_t)by * (uint64_t)z);
            oct[b] = ow;
            lng[b] = lw;
            uint32_t D = least;
            if (least == (uint32_t)kCap) {
                if (FAR == FarBricks::kNone) D = kMaxBrickDistance;
                if (FAR == FarBricks::kHere) D = direct_distance(s.rows[0], x, y, z, by, bz, row_words(bx));
                far = FAR != FarBricks::kNone;
            }
            if (least) dir[b] = kEmptyBit | D;
        }
    }
    if (far) *s.deep = 1u;
}

// Axes y and z: long-box words, from the octant words.
template <int A>
__device__ __forceinline__ void lattice_long(const LatticeScratch& s,
                                             const uint32_t* __restrict__ oct,
                                             uint32_t* __restrict__ lng, int32_t bx, int32_t by,
                                             int32_t bz, const BrickBox& w, uint32_t tile,
                                             uint64_t* tab) {
    uint64_t* lev = tab + kTableWords;
    const Tile t = lattice_tile<A>(w, tile, bx, by, bz);
    // the tile's octant words, 8 bricks along x at a time (32-byte pieces); the brick a0 + a of row
    // (c1, c2) is (t1 + c1, a0 + a, t2 + c2) for A = 1 and (t1 + c1, t2 + c2, a0 + a) for A = 2
    const int32_t ea = (A == 1 ? w.y0 + w.ny : w.z0 + w.nz), e1 = w.x0 + w.nx,
                  e2 = (A == 1 ? w.z0 + w.nz : w.y0 + w.ny);
    const int32_t c1 = (int32_t)(threadIdx.x & 7u), a = (int32_t)((threadIdx.x >> 3) & 31u);
    const bool mine = t.a0 + a < ea && t.t1 + c1 < e1;
    const uint64_t plane = (uint64_t)bx * by;
    const uint64_t b0 = (uint64_t)(t.t1 + c1) + (A == 1 ? (uint64_t)bx * (uint64_t)(t.a0 + a) + plane * (uint64_t)t.t2
                                                        : plane * (uint64_t)(t.a0 + a) + (uint64_t)bx * (uint64_t)t.t2);
    const uint64_t step2 = A == 1 ? plane : (uint64_t)bx;
    uint32_t ow[kTile];
#pragma unroll
    for (int32_t c2 = 0; c2 < kTile; ++c2)
        ow[c2] = mine && t.t2 + c2 < e2 ? __ldg(oct + b0 + step2 * (uint64_t)c2) : 0u;
    lattice_tables(s.rows[A], t, tab);
    {
        const int32_t row = threadIdx.x & (kRows - 1), q = threadIdx.x / kRows;
        const int32_t at = ((row / kTile) + kHalo) * kPitch + (row % kTile) + kHalo;
        const int32_t n1 = (q & 1) ? -1 : 0, n2 = (q & 2) ? -1 : 0;
#pragma unroll
        for (int k = 1; k <= kCap; ++k)
            lev[(k - 1) * kLevelPitch + q * kRows + row] = merged_row(tab, at, n1, n2, k);
    }
    __syncthreads();  // the tables are read: their space takes the words, turned to lanes along A
    uint32_t* turn = reinterpret_cast<uint32_t*>(tab);  // [row][33]
#pragma unroll
    for (int32_t c2 = 0; c2 < kTile; ++c2) turn[(c2 * kTile + c1) * 33 + a] = ow[c2];
    __syncthreads();
    const uint32_t lane = threadIdx.x & 31u;
#pragma unroll 2
    for (int32_t r = (int32_t)(threadIdx.x >> 5); r < kRows; r += kLatticeThreads / 32) {
        const uint32_t o_w = turn[r * 33 + lane];
        uint32_t lw = 0;
#pragma unroll
        for (int o = 0; o < 8; ++o) {
            const uint32_t K = (o_w >> (4 * o)) & 15u;
            // lateral signs in ascending axis order: (x, z) for A = 1, (x, y) for A = 2
            const int qo = A == 1 ? ((o & 1) | ((o >> 1) & 2)) : (o & 3);
            const uint64_t m = lev[(max(K, 1u) - 1u) * kLevelPitch + qo * kRows + r];
            lw |= (((o >> A) & 1) ? run_backward(m, lane) : run_forward(m, lane)) << (4 * o);
        }
        turn[r * 33 + lane] = lw;
    }
    __syncthreads();
    uint32_t* out = lng + (uint64_t)A * ((uint64_t)bx * by * bz) + b0;
#pragma unroll
    for (int32_t c2 = 0; c2 < kTile; ++c2)
        if (mine && t.t2 + c2 < e2) out[step2 * (uint64_t)c2] = turn[(c2 * kTile + c1) * 33 + a];
}

__global__ void __launch_bounds__(kLatticeThreads) lattice_yz_kernel(
    LatticeScratch s, const uint32_t* __restrict__ oct, uint32_t* __restrict__ lng, int32_t bx,
    int32_t by, int32_t bz, BrickBox w, uint32_t tiles_y) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    uint64_t* tab = reinterpret_cast<uint64_t*>(smem_raw);
    if (blockIdx.x < tiles_y)
        lattice_long<1>(s, oct, lng, bx, by, bz, w, blockIdx.x, tab);
    else
        lattice_long<2>(s, oct, lng, bx, by, bz, w, blockIdx.x - tiles_y, tab);
}

// ---------------------------------------------------------------------------------------------
// Distances of bricks with no occupied brick within 14 (all of them, with oct == nullptr): the
// separable transform.  Pass xy takes, per brick, the minimum over rows y' of max(|y' - y|, distance
// along x in row y') from the x rows (two word reads and a find-first-set per side); pass z the
// minimum over z' of max(|z' - z|, pass xy).  Both walk outward and stop once the offset reaches the
// best value found.
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ bool box_brick(const BrickBox& box, int32_t bx, int32_t by, int32_t& x,
                                          int32_t& y, int32_t& z, uint64_t& b) {
    const uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (uint64_t)box.nx * box.ny * box.nz) return false;
    x = box.x0 + (int32_t)(t % (uint64_t)box.nx);
    const uint64_t r = t / (uint64_t)box.nx;
    y = box.y0 + (int32_t)(r % (uint64_t)box.ny);
    z = box.z0 + (int32_t)(r / (uint64_t)box.ny);
    b = (uint64_t)x + (uint64_t)bx * ((uint64_t)y + (uint64_t)by * (uint64_t)z);
    return true;
}

__global__ void __launch_bounds__(256) lattice_distance_xy_kernel(const uint32_t* __restrict__ rows,
                                                                  uint8_t* __restrict__ out,
                                                                  int32_t bx, int32_t by,
                                                                  BrickBox box) {
    int32_t x, y, z;
    uint64_t b;
    if (!box_brick(box, bx, by, x, y, z, b)) return;
    const int32_t rw = row_words(bx);
    const uint32_t* plane = rows + (uint64_t)z * by * rw;
    int32_t best = (int32_t)kMaxBrickDistance;
    for (int32_t r = 0; r < best; ++r) {
        if (y + r < by) best = min(best, max(r, row_distance(plane + (uint64_t)(y + r) * rw, rw, x, (int32_t)kMaxBrickDistance)));
        if (r && y - r >= 0) best = min(best, max(r, row_distance(plane + (uint64_t)(y - r) * rw, rw, x, (int32_t)kMaxBrickDistance)));
    }
    out[b] = (uint8_t)best;
}

__global__ void __launch_bounds__(256) lattice_distance_z_kernel(uint32_t* __restrict__ dir,
                                                                 const uint32_t* __restrict__ oct,
                                                                 const uint8_t* __restrict__ in,
                                                                 int32_t bx, int32_t by, int32_t bz,
                                                                 BrickBox box) {
    int32_t x, y, z;
    uint64_t b;
    if (!box_brick(box, bx, by, x, y, z, b)) return;
    if (oct ? oct[b] != 0xFFFFFFFFu : !brick_empty(dir[b])) return;
    const uint64_t plane = (uint64_t)bx * by;
    int32_t best = (int32_t)kMaxBrickDistance;
    for (int32_t r = 0; r < best; ++r) {
        if (z + r < bz) best = min(best, max(r, (int32_t)__ldg(in + b + plane * (uint64_t)r)));
        if (r && z - r >= 0) best = min(best, max(r, (int32_t)__ldg(in + b - plane * (uint64_t)r)));
    }
    dir[b] = kEmptyBit | (uint32_t)max(best, 1);
}

// ---------------------------------------------------------------------------------------------

static inline size_t align16(size_t v) { return (v + 15) / 16 * 16; }

static size_t row_bytes(int32_t na, uint64_t rows) { return align16((size_t)((na + 31) / 32) * rows * 4); }

size_t lattice_scratch_bytes(int32_t bx, int32_t by, int32_t bz) {
    return row_bytes(bx, (uint64_t)by * bz) + row_bytes(by, (uint64_t)bx * bz) +
           row_bytes(bz, (uint64_t)bx * by) + align16((size_t)bx * by * bz) + 16;
}

LatticeScratch carve_lattice_scratch(void* base, int32_t bx, int32_t by, int32_t bz) {
    char* p = (char*)base;
    LatticeScratch s;
    s.deep = (uint32_t*)p;
    p += 16;
    s.rows[0] = (uint32_t*)p;
    p += row_bytes(bx, (uint64_t)by * bz);
    s.rows[1] = (uint32_t*)p;
    p += row_bytes(by, (uint64_t)bx * bz);
    s.rows[2] = (uint32_t*)p;
    p += row_bytes(bz, (uint64_t)bx * by);
    s.dist = (uint8_t*)p;
    return s;
}

// `b` grown by g bricks on each side (gx along x, ...), clipped to the lattice.
static BrickBox grow(const BrickBox& b, int32_t gx, int32_t gy, int32_t gz, int32_t bx, int32_t by,
                     int32_t bz) {
    BrickBox r;
    r.x0 = max(b.x0 - gx, 0);
    r.y0 = max(b.y0 - gy, 0);
    r.z0 = max(b.z0 - gz, 0);
    r.nx = min(b.x0 + b.nx + gx, bx) - r.x0;
    r.ny = min(b.y0 + b.ny + gy, by) - r.y0;
    r.nz = min(b.z0 + b.nz + gz, bz) - r.z0;
    return r;
}

// The smallest box of whole 32-brick words around `b`.
static BrickBox word_box(const BrickBox& b, int32_t bx, int32_t by, int32_t bz) {
    BrickBox r;
    r.x0 = b.x0 & ~31;
    r.y0 = b.y0 & ~31;
    r.z0 = b.z0 & ~31;
    r.nx = min((b.x0 + b.nx + 31) & ~31, bx) - r.x0;
    r.ny = min((b.y0 + b.ny + 31) & ~31, by) - r.y0;
    r.nz = min((b.z0 + b.nz + 31) & ~31, bz) - r.z0;
    return r;
}

static void launch_rows(const uint32_t* dir, const LatticeScratch& s, int32_t bx, int32_t by,
                        int32_t bz, const BrickBox& need, cudaStream_t stream) {
    const BrickBox b = word_box(need, bx, by, bz);
    const uint64_t wx = (uint64_t)(b.nx + 31) / 32, wy = (uint64_t)(b.ny + 31) / 32, wz = (uint64_t)(b.nz + 31) / 32;
    const uint64_t warps = wx * wy * (uint64_t)b.nz + wx * (uint64_t)b.ny * wz;
    lattice_rows_kernel<<<(unsigned)((warps + 7) / 8), 256, 0, stream>>>(dir, s, bx, by, bz, b);
}

static unsigned tiles(int32_t na, int32_t n1, int32_t n2) {
    return (unsigned)((uint64_t)((na + 31) / 32) * ((n1 + kTile - 1) / kTile) * ((n2 + kTile - 1) / kTile));
}

cudaError_t launch_brick_lattice(uint32_t* dir, uint32_t* oct, uint32_t* lng,
                                 const LatticeScratch& s, int32_t bx, int32_t by, int32_t bz,
                                 cudaStream_t stream, const BrickBox* changed) {
    // above 48 KiB of dynamic shared memory: opted in on every call (cheap), so that a re-created
    // context has it too
    auto* x_kernel = lattice_x_kernel<FarBricks::kLater>;
    if (std::max({bx, by, bz}) <= kCap)
        x_kernel = lattice_x_kernel<FarBricks::kNone>;
    else if (!changed && (uint64_t)bx * by * bz <= kDirectBricks)  // (after a change not all rows are there)
        x_kernel = lattice_x_kernel<FarBricks::kHere>;
    cudaError_t e = cudaFuncSetAttribute((const void*)x_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)kLatticeShared);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute((const void*)lattice_yz_kernel,
                                 cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kLatticeShared);
    if (e != cudaSuccess) return e;
    const BrickBox all = {0, 0, 0, bx, by, bz};
    // a box from a brick reaches 14 bricks past it, so a change reaches 14 bricks back; the words
    // there read rows up to 14 further out
    const BrickBox w = changed ? grow(*changed, kHalo, kHalo, kHalo, bx, by, bz) : all;
    launch_rows(dir, s, bx, by, bz, changed ? grow(w, kCap, kCap, kCap, bx, by, bz) : all, stream);
    x_kernel<<<tiles(w.nx, w.ny, w.nz), kLatticeThreads, kLatticeShared, stream>>>(s, dir, oct, lng, bx, by, bz, w);
    const unsigned ty = tiles(w.ny, w.nx, w.nz), tz = tiles(w.nz, w.nx, w.ny);
    lattice_yz_kernel<<<ty + tz, kLatticeThreads, kLatticeShared, stream>>>(s, oct, lng, bx, by, bz, w, ty);
    return cudaGetLastError();
}

cudaError_t launch_brick_distance(uint32_t* dir, const uint32_t* oct, const LatticeScratch& s,
                                  int32_t bx, int32_t by, int32_t bz, cudaStream_t stream,
                                  const BrickBox* changed) {
    // distances change only within 31 bricks of a change; pass z reads pass xy up to 31 bricks away
    // along z, which reads the x rows up to 31 away along y
    const int32_t R = (int32_t)kMaxBrickDistance;
    const BrickBox all = {0, 0, 0, bx, by, bz};
    const BrickBox w = changed ? grow(*changed, R, R, R, bx, by, bz) : all;
    const BrickBox w1 = grow(w, 0, 0, R, bx, by, bz);
    if (!oct || changed)  // the rows of launch_brick_lattice reach less far
        launch_rows(dir, s, bx, by, bz, grow(w1, R, R, 0, bx, by, bz), stream);
    auto blocks = [](const BrickBox& b) { return (unsigned)(((uint64_t)b.nx * b.ny * b.nz + 255) / 256); };
    lattice_distance_xy_kernel<<<blocks(w1), 256, 0, stream>>>(s.rows[0], s.dist, bx, by, w1);
    lattice_distance_z_kernel<<<blocks(w), 256, 0, stream>>>(dir, oct, s.dist, bx, by, bz, w);
    return cudaGetLastError();
}

}  // namespace vt
