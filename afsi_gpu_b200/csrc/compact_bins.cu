// Compact spread with the markers binned first.
//
// Marker clouds come in no order, so the plain compact spread (transfer.cu)
// reduces every point's 64 links into the L2: 28 sectors per point and
// component, at the L2's 110 G sector reductions/s.  Where many markers share a
// lattice cell most of those reductions meet in the same faces.  Here the points
// are ordered by 4x4x4-cell tile and cell (a count per cell, a scan, a place per
// point), a warp takes 32 consecutive points and sums each component into a box
// in shared memory, and each face of the box is reduced once.  A box that covers
// all of the warp's points is used where it fits, else the points go tile by
// tile: a tile's box is at most 8x8x8 faces (four cells, one more where the
// component's lattice is shifted, three of overhang).  Points that share their
// support origin (kBinMerge and more per origin) are summed first (FP64 tensor
// cores, runs.cuh), others are added one by one; few points of a tile are reduced
// directly.
//
// What bounds it is latency at 20 warps per SM (96 registers, 9.5 KB of shared
// memory a warp; issue 47 %), first of all the scattered reads of the table rows.  Lanes
// therefore read whole rows together (cp.async, 16 bytes each), the bases and
// forces of all components are requested at once, and the next component's rows
// are in flight while a box is flushed: 186 -> 138 us; 32 points per warp at 20
// warps instead of 64 at 16: 123 us (24 warps: 127).  400,000 markers of a shell on
// 64^3 (50 per cell), FP64, one B200: 305 us plain, 123 us and 36 us of binning and
// clearing here.  The caller chooses the form by the cloud's density
// (bin_density_kernel, cuda_ib.compact_spread).
#include <cub/device/device_scan.cuh>
#include <climits>
#include <cmath>
#include "common.cuh"
#include "runs.cuh"

namespace afsi {
namespace {

constexpr int kBinWarps = 4;
constexpr int kBinPoints = 32;    // points per warp
constexpr int kBinCap = 608;      // padded 8x8x8 box
constexpr int kBinMerge = 3;      // points per run from which the runs are summed first
constexpr int kBinOut = 0xffff;
constexpr int kBinFew = 4;        // fewer points of a tile than this are reduced directly

struct BinGrid {
    int nx, ny, nz;        // cells
    int t1, t2;            // tiles along y and z
    unsigned none;         // key of points without a tile
};

__device__ __forceinline__ int bin_extent(const BinGrid& g, int c, int a) {
    return (a == 0 ? g.nx : a == 1 ? g.ny : g.nz) + (a == c);
}

__device__ __forceinline__ unsigned bin_key(int64_t x, int64_t y, int64_t z, const BinGrid& g) {
    if (!(x >= 0 && y >= 0 && z >= 0 && x <= g.nx - 3 && y < g.ny - 3 && z < g.nz - 3)) return g.none;
    const int ix = int(x), iy = int(y), iz = int(z);
    return unsigned(((ix >> 2) * g.t1 + (iy >> 2)) * g.t2 + (iz >> 2)) * 64u +
           unsigned(((ix & 3) << 4) | ((iy & 3) << 2) | (iz & 3));
}

// Cell of component 0's support origin (tile * 64 + cell of the tile) and the
// point's rank among the points of that cell.
__global__ void __launch_bounds__(256) bin_count_kernel(const int64_t* __restrict__ base, int64_t points, BinGrid g,
                                                        int32_t* __restrict__ count, uint2* __restrict__ place) {
    const int64_t p = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (p >= points) return;
    const unsigned key = bin_key(base[p * 3], base[p * 3 + 1], base[p * 3 + 2], g);
    place[p] = make_uint2(key, unsigned(atomicAdd(count + key, 1)));
}

__global__ void __launch_bounds__(256) bin_order_kernel(const uint2* __restrict__ place,
                                                        const int32_t* __restrict__ first, int64_t points,
                                                        int32_t* __restrict__ order) {
    const int64_t p = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (p >= points) return;
    const uint2 k = place[p];
    order[first[k.x] + int32_t(k.y)] = int32_t(p);
}

// Points per occupied cell, by a sample: one block takes kSample points at even
// distances and counts those that find their cell (component 0's support origin)
// taken by an earlier one.  More than `limit` of them set `bit` of the status word.
constexpr int kSample = 4096, kSampleSlots = 2 * kSample;
__global__ void __launch_bounds__(1024) bin_density_kernel(const int64_t* __restrict__ base, int64_t points, int limit,
                                                           int32_t bit, int32_t* status) {
    __shared__ unsigned slot[kSampleSlots];
    constexpr unsigned kFree = 0xffffffffu;
    for (int i = threadIdx.x; i < kSampleSlots; i += 1024) slot[i] = kFree;
    __syncthreads();
    int again = 0;
#pragma unroll
    for (int k = 0; k < kSample / 1024; ++k) {
        const int64_t p = (int64_t(threadIdx.x) + 1024 * k) * points / kSample;
        const int64_t x = base[p * 3], y = base[p * 3 + 1], z = base[p * 3 + 2];
        if (x < 0 || y < 0 || z < 0 || ((x | y | z) >> 20)) continue;
        // 31 mixed bits stand for the cell (one pair in 2^31 is mistaken)
        const uint64_t cell = uint64_t(x) << 40 | uint64_t(y) << 20 | uint64_t(z);
        const unsigned key = unsigned((cell * 0x9e3779b97f4a7c15ull) >> 33);
        unsigned h = key;
        for (int t = 0; t < kSampleSlots; ++t, ++h) {  // at most kSample slots are taken
            const unsigned old = atomicCAS(&slot[h % kSampleSlots], kFree, key);
            if (old == kFree) break;
            if (old == key) {
                ++again;
                break;
            }
        }
    }
    again = int(__reduce_add_sync(0xffffffffu, unsigned(again)));
    __shared__ int total;
    if (threadIdx.x == 0) total = 0;
    __syncthreads();
    if ((threadIdx.x & 31) == 0) atomicAdd(&total, again);
    __syncthreads();
    if (threadIdx.x == 0 && total > limit) atomicOr(status, bit);
}

template <class T>
struct __align__(16) BinStage {
    T w[(kBinPoints + 1) * 12];  // rows of the component; the last stays zero
    T box[kBinCap];
    T f[kBinPoints + 1];         // force / volume; the last stays zero
    int id[kBinPoints], key[kBinPoints], rk[kBinPoints];
    uint16_t b[3][kBinPoints * 3];  // support origins; kBinOut: negative or too large
    uint16_t rs[kBinPoints + 1];
    uint8_t perm[4 * kBinPoints];
};

// Weight rows of component c of the warp's n points into s.w: 16 bytes per lane
// and copy, so the lanes of a copy read whole rows of five or ten points.
template <class T>
__device__ __forceinline__ void bin_fetch_rows(BinStage<T>& s, const T* __restrict__ phi, int64_t points, int c, int n) {
    constexpr int K = 12 * int(sizeof(T)) / 16;  // copies per point
    for (int t = threadIdx.x & 31; t < n * K; t += 32) {
        const int q = t / K;
        const T* src = phi + (c * points + s.id[q]) * 12 + (t - q * K) * (16 / int(sizeof(T)));
        const unsigned dst = static_cast<unsigned>(__cvta_generic_to_shared(s.w)) + unsigned(t) * 16u;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
    }
}

// Adds the points with at[q] >= 0 (offset of the support origin) one after
// another: lane (h, i, j) adds z links 2h and 2h + 1 of the link column (i, j); the
// next point's weights are read before this point's sums are written.
template <class T>
__device__ __forceinline__ void bin_points(T* box, const int* at, const T* f, const T* w, int n, int sx, int sy) {
    using P = typename std::conditional<sizeof(T) == 8, double2, float2>::type;
    const int lane = threadIdx.x & 31, half = lane >> 4, li = (lane >> 2) & 3, lj = lane & 3;
    T* const mine = box + li * sx + lj * sy + 2 * half;
    int k = at[0];
    T a = (w[li] * w[4 + lj]) * f[0];
    P z = reinterpret_cast<const P*>(w + 8)[half];
    for (int q = 1; q <= n; ++q) {  // row n lies inside the arrays
        const int kn = q < n ? at[q] : -1;
        const T* row = w + q * 12;
        const T wx = row[li], wy = row[4 + lj], fn = f[q];
        const P zn = reinterpret_cast<const P*>(row + 8)[half];
        if (k >= 0) {
            T* dst = mine + k;
            const T t0 = dst[0], t1 = dst[1];
            dst[0] = fma(a, z.x, t0);
            dst[1] = fma(a, z.y, t1);
        }
        __syncwarp();
        k = kn;
        a = (wx * wy) * fn;
        z = zn;
    }
}

template <class T>
__global__ void __launch_bounds__(kBinWarps * 32, 5) bin_spread_kernel(
    const T* __restrict__ force, const int64_t* __restrict__ base, const T* __restrict__ phi, int64_t points,
    const int32_t* __restrict__ order, BinGrid g, T volume, T inv_volume,
    T* __restrict__ u0, T* __restrict__ u1, T* __restrict__ u2, int32_t* status) {
    extern __shared__ __align__(16) unsigned char bin_smem[];
    BinStage<T>& s = reinterpret_cast<BinStage<T>*>(bin_smem)[threadIdx.x >> 5];
    static_assert(kBinPoints == 32, "a point per lane");
    const int lane = threadIdx.x & 31;
    const int64_t chunk = int64_t(blockIdx.x) * kBinWarps + (threadIdx.x >> 5), q0 = chunk * kBinPoints;
    if (q0 >= points) return;  // whole warp
    const int n = int(points - q0 < kBinPoints ? points - q0 : kBinPoints);
    if (lane < 12) s.w[kBinPoints * 12 + lane] = T(0);
    if (lane == 0) s.f[kBinPoints] = T(0);
    const bool mine = lane < n;
    s.id[lane] = mine ? order[q0 + lane] : 0;
    __syncwarp();
    bin_fetch_rows(s, phi, points, 0, n);
    T force_of[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) force_of[c] = mine ? force[int64_t(s.id[lane]) * 3 + c] : T(0);
#pragma unroll
    for (int i = 0; i < 9; ++i) {  // 3 components, 3 rounds of 32 coordinates
        const int c = i / 3, t = lane + 32 * (i - c * 3), q = t / 3;
        const int64_t v = q < n ? base[(c * points + s.id[q]) * 3 + (t - 3 * q)] : -1;
        s.b[c][t] = v >= 0 && v < kBinOut ? uint16_t(v) : kBinOut;
    }
    __syncwarp();
    const uint16_t* b0 = s.b[0] + lane * 3;
    const unsigned cell = bin_key(b0[0], b0[1], b0[2], g), tile = cell == g.none ? 0xfffffffeu : cell >> 6;
#pragma unroll 1
    for (int c = 0; c < 3; ++c) {
        T* field = c == 0 ? u0 : c == 1 ? u1 : u2;
        const int e0 = bin_extent(g, c, 0), e1 = bin_extent(g, c, 1), e2 = bin_extent(g, c, 2);
        int b[3];
#pragma unroll
        for (int a = 0; a < 3; ++a) b[a] = s.b[c][lane * 3 + a];
        const bool live = mine && b[0] + 3 < e0 && b[1] + 3 < e1 && b[2] + 3 < e2;
        if (mine && !live) flag(status, AFSI_FLAG_INDEX);
        const T fv = c == 0 ? force_of[0] : c == 1 ? force_of[1] : force_of[2];
        if (mine) s.f[lane] = inv_volume != T(0) ? fv * inv_volume : fv / volume;
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncwarp();
        // the whole warp at once when one box covers it, else tile by tile
        bool left = live, whole = true, fetched = c == 2;  // fetched: the next component's rows
        while (true) {
            const unsigned rest = __ballot_sync(0xffffffffu, left);
            if (!rest) {
                if (!fetched) bin_fetch_rows(s, phi, points, c + 1, n);  // no point of this component
                break;
            }
            const unsigned now = __shfl_sync(0xffffffffu, tile, __ffs(rest) - 1);  // the tile of a point that is left
            const bool take = left && (whole || tile == now);
            int mn[3], mx[3];
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                mn[a] = __reduce_min_sync(0xffffffffu, take ? b[a] : INT_MAX);
                mx[a] = __reduce_max_sync(0xffffffffu, take ? b[a] : INT_MIN);
            }
            left = left && !take;
            const int ex = mx[0] - mn[0] + 4, ey = mx[1] - mn[1] + 4, ez = mx[2] - mn[2] + 4;
            int sx = 0, sy = 0;
            bool fits = ey <= 64 && ez <= 64;
            if (fits) {
                padded_strides(ey, ez, sx, sy);
                fits = int64_t(ex) * sx <= kBinCap;
            }
            if (whole && !fits) {
                whole = false;
                left = live;
                continue;
            }
            const unsigned taken = __ballot_sync(0xffffffffu, take);
            const int count = __popc(taken);
            const bool fetch = !fetched && !__any_sync(0xffffffffu, left);
            fetched = fetched || fetch;
            if (fits && count >= kBinFew) {
                const int size = ex * sx;
                for (int t = lane; t < size; t += 32) s.box[t] = T(0);
                const int d0 = b[0] - mn[0], d1 = b[1] - mn[1], d2 = b[2] - mn[2];
                int key = take ? run_key(d0, d1, d2) : -1;
                const unsigned peers = __match_any_sync(0xffffffffu, key);
                const int runs = __popc(__ballot_sync(0xffffffffu, take && (peers & ((1u << lane) - 1u)) == 0u));
                const bool merge = count >= kBinMerge * runs;
                if (!merge && take) key = d0 * sx + d1 * sy + d2;
                s.key[lane] = key;
                __syncwarp();
                if (merge)
                    spread_element<T, kBinPoints>(s.box, s.key, s.f, s.w, s.w + 4, s.w + 8, n, sx, sy, s.perm, s.rs,
                                                  s.rk);
                else
                    bin_points(s.box, s.key, s.f, s.w, n, sx, sy);
                __syncwarp();
                if (fetch) bin_fetch_rows(s, phi, points, c + 1, n);
                const int cells = ex * ey * ez, qz = 32 % ez, r = 32 / ez, qy = r % ey, qx = r / ey;
                int z = lane % ez, t = lane / ez, y = t % ey, x = t / ey;
                for (int k = lane; k < cells; k += 32) {
                    const int o = x * sx + y * sy + z;
                    const T v = s.box[o];
                    if (v != T(0))
                        atomicAdd(field + (int64_t(mn[0] + x) * e1 + (mn[1] + y)) * e2 + (mn[2] + z), v);
                    z += qz;
                    int carry = z >= ez ? 1 : 0;
                    z -= carry * ez;
                    y += qy + carry;
                    carry = y >= ey ? 1 : 0;
                    y -= carry * ey;
                    x += qx + carry;
                }
                __syncwarp();
            } else {  // four lanes per point, lane k on z link k, as the plain form
                __syncwarp();
                for (unsigned todo = taken; todo;) {  // up to eight points at a time
                    unsigned next = todo;
                    for (int k = 0; k < (lane >> 2) && next; ++k) next &= next - 1;
                    const bool has = next != 0;
                    const int src = has ? __ffs(next) - 1 : 0;
                    const int bx = __shfl_sync(0xffffffffu, b[0], src), by = __shfl_sync(0xffffffffu, b[1], src),
                              bz = __shfl_sync(0xffffffffu, b[2], src);
                    if (has) {
                        const T* w = s.w + src * 12;
                        const int k = lane & 3;
                        const T fz = s.f[src] * w[8 + k];
                        T* dst = field + (int64_t(bx) * e1 + by) * e2 + bz + k;
                        for (int i = 0; i < 4; ++i)
                            for (int l = 0; l < 4; ++l)
                                atomicAdd(dst + (int64_t(i) * e1 + l) * e2, (w[i] * w[4 + l]) * fz);
                    }
                    for (int k = 0; k < 8 && todo; ++k) todo &= todo - 1;
                }
                __syncwarp();
                if (fetch) bin_fetch_rows(s, phi, points, c + 1, n);
            }
        }
    }
}

inline int64_t bin_slab(int64_t bytes) { return (bytes + 255) / 256 * 256; }

inline int64_t bin_tiles(int64_t nx, int64_t ny, int64_t nz) {
    return ((nx + 1 + 3) / 4) * ((ny + 3) / 4) * ((nz + 3) / 4);
}

size_t bin_scan_bytes(int64_t cells) {
    size_t t = 0;
    cub::DeviceScan::ExclusiveSum(nullptr, t, static_cast<const int32_t*>(nullptr), static_cast<int32_t*>(nullptr),
                                  cells);
    return t;
}

}  // namespace
}  // namespace afsi

using namespace afsi;

extern "C" int64_t afsi_b200_compact_binned_bytes(int64_t points, int64_t nx, int64_t ny, int64_t nz) {
    if (points < 0 || points >= INT32_MAX || nx < 1 || ny < 1 || nz < 1 || nx >= kBinOut - 4 || ny >= kBinOut - 4 ||
        nz >= kBinOut - 4 || bin_tiles(nx, ny, nz) >= (int64_t(1) << 26))
        return -1;
    const int64_t cells = bin_tiles(nx, ny, nz) * 64 + 64;  // one tile more for the points without a cell
    return bin_slab(points * 8) + bin_slab(points * 4) + 2 * bin_slab(cells * 4) + bin_slab(bin_scan_bytes(cells));
}

extern "C" int32_t afsi_b200_compact_spread3_binned(const void* force, const int64_t* base, const void* phi,
                                                    int64_t points, int64_t nx, int64_t ny, int64_t nz, double volume,
                                                    void* u0, void* u1, void* u2, void* scratch, int64_t scratch_bytes,
                                                    int32_t* status, int32_t dtype, afsi_stream_t stream) {
    AFSI_REQUIRE(nx > 0 && ny > 0 && nz > 0 && points >= 0, "invalid compact grid");
    AFSI_REQUIRE(isfinite(volume) && volume > 0, "invalid compact grid/volume");
    AFSI_REQUIRE(u0 && u1 && u2, "null device pointer");
    const int64_t need = afsi_b200_compact_binned_bytes(points, nx, ny, nz);
    AFSI_REQUIRE(need >= 0, "too many points or tiles for the binned spread");
    const size_t es = dtype == AFSI_F64 ? 8 : 4;
    if (cudaMemsetAsync(u0, 0, size_t((nx + 1) * ny * nz) * es, stream) != cudaSuccess ||
        cudaMemsetAsync(u1, 0, size_t(nx * (ny + 1) * nz) * es, stream) != cudaSuccess ||
        cudaMemsetAsync(u2, 0, size_t(nx * ny * (nz + 1)) * es, stream) != cudaSuccess)
        return fail(AFSI_ERR_CUDA, "clearing the face arrays failed");
    if (points == 0) return AFSI_OK;
    AFSI_REQUIRE(force && base && phi && scratch, "null device pointer");
    AFSI_REQUIRE(reinterpret_cast<uintptr_t>(phi) % 16 == 0, "the binned spread needs 16-byte aligned weights");
    AFSI_REQUIRE(scratch_bytes >= need, "binned spread scratch too small");
    const int64_t tiles = bin_tiles(nx, ny, nz), cells = tiles * 64 + 64;
    unsigned char* m = static_cast<unsigned char*>(scratch);
    uint2* place = reinterpret_cast<uint2*>(m);
    int32_t* order = reinterpret_cast<int32_t*>(m += bin_slab(points * 8));
    int32_t* count = reinterpret_cast<int32_t*>(m += bin_slab(points * 4));
    int32_t* first = reinterpret_cast<int32_t*>(m += bin_slab(cells * 4));
    void* temp = m += bin_slab(cells * 4);
    size_t temp_bytes = bin_scan_bytes(cells);
    const BinGrid g{int(nx), int(ny), int(nz), int((ny + 3) / 4), int((nz + 3) / 4), unsigned(tiles * 64)};
    if (cudaMemsetAsync(count, 0, size_t(cells) * 4, stream) != cudaSuccess)
        return fail(AFSI_ERR_CUDA, "clearing the bin counts failed");
    bin_count_kernel<<<blocks_for(points, 256), 256, 0, stream>>>(base, points, g, count, place);
    int32_t rc = launched("compact bin counts");
    if (rc) return rc;
    if (cub::DeviceScan::ExclusiveSum(temp, temp_bytes, count, first, cells, stream) != cudaSuccess)
        return fail(AFSI_ERR_CUDA, "compact bin scan failed");
    bin_order_kernel<<<blocks_for(points, 256), 256, 0, stream>>>(place, first, points, order);
    rc = launched("compact bin order");
    if (rc) return rc;
    AFSI_DISPATCH(dtype, {
        const T vol = T(volume);
        const size_t smem = sizeof(BinStage<T>) * kBinWarps;
        if ((rc = allow_shared<bin_spread_kernel<T>>("compact_spread3_binned", smem))) return rc;
        const int64_t warps = (points + kBinPoints - 1) / kBinPoints;
        bin_spread_kernel<T><<<blocks_for(warps, kBinWarps), kBinWarps * 32, smem, stream>>>(
            static_cast<const T*>(force), base, static_cast<const T*>(phi), points, order, g, vol, exact_inverse(vol),
            static_cast<T*>(u0), static_cast<T*>(u1), static_cast<T*>(u2), status);
    });
    return launched("compact_spread3_binned");
}

extern "C" int32_t afsi_b200_compact_density(const int64_t* base, int64_t points, double per_cell, int32_t bit,
                                             int32_t* status, afsi_stream_t stream) {
    AFSI_REQUIRE(points >= 0 && per_cell > 0 && isfinite(per_cell), "invalid compact density question");
    if (points < kSample) return AFSI_OK;
    AFSI_REQUIRE(base && status, "null device pointer");
    // points that meet an earlier one among kSample points in `cells` equally likely cells
    const double cells = double(points) / per_cell;
    const int limit = int(kSample - cells * (1.0 - std::exp(-kSample / cells)));
    bin_density_kernel<<<1, 1024, 0, stream>>>(base, points, limit, bit, status);
    return launched("compact_density");
}
