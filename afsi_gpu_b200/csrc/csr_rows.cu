// P1 CSR operators built row by row (no hash table).
//
// B_c[node, face] = Σ over the cells holding the node, Σ over the cell's
// points of W·N[q,a]·φx·φy·φz (mac/assembled_transfer.py:151-216).  The hash
// contraction (csr.cu) adds every (cell, node, face) sum into a table at random
// addresses and then sorts the table; here the rows are formed directly:
//
//   boxes      per element and component the box of its points' supports, and
//              the (node, slot) pairs of the connectivity (slot = 4 e + a);
//   incidence  the pairs sorted by node (stable, so a node's cells keep their
//              order), per node and component the union of its cells' boxes and,
//              by one scan of the box volumes, the row's place in a padded buffer
//              shared by the three components;
//   fill       one warp per (component, node): the union box in shared memory,
//              the points of the node's cells in order (32 points staged at a
//              time, whichever cells they belong to): FP64 sums the points of
//              one support origin on the tensor cores (spread_runs_mma) and
//              adds each sum, FP32 adds point by point;
//              the touched entries leave the box in ascending face order, which
//              is the CSR column order: B needs no sort.  An entry exists when
//              something nonzero was added to it (untouched entries hold -0, which
//              no sum of nonzero terms gives): in FP32 a point's product, in FP64
//              the sum of one origin's points among the 32 staged, in the hash
//              form a cell's sum.  The three differ where contributions of either
//              sign cancel exactly, and then in explicit zeros;
//   finish     the padded rows packed to CSR, and the transpose by a stable
//              radix sort on the face index alone (32-bit keys and positions).
//
// No atomics on values: the operators are the same bit for bit on every run.
// What bounds it: the fill is bound by the L1's data stage (73 %; 64 links per
// point and component added in shared memory, each cell visited by its four nodes;
// adding every point by itself kept it 80 % busy), the finish by the HBM passes of
// the sort.  128,000 tetrahedra (1.2 M points) on 128^3, FP64, one B200: fill
// 0.78 ms (1.04 ms point by point), sorts 0.39 ms, pack and transpose 0.29 ms
// for the three components, where the hash contraction took 4.98 ms and the
// table's sorts 2.57 ms; tables, assembly, spread and interpolate together
// 9.64 -> 2.38 ms.
#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_scan.cuh>
#include <algorithm>
#include "common.cuh"
#include "runs.cuh"

namespace afsi {
namespace {

constexpr int kRowsWarps = 4;    // warps (rows) per block of the fill
constexpr int kRowsGroups = AFSI_ROWS_GROUPS;
constexpr int kMaxExt = 1023;    // packed box extents: 10 bits each

struct FaceDims {
    int nx, ny, nz;  // cells
};

__host__ __device__ __forceinline__ int face_n(const FaceDims& g, int c, int a) {
    return (a == 0 ? g.nx : a == 1 ? g.ny : g.nz) + (a == c);
}

// Box of a support set: lower corner and extents (0: empty).
__device__ __forceinline__ int4 pack_box(const int mn[3], const int mx[3]) {
    return make_int4(mn[0], mn[1], mn[2],
                     (mx[0] - mn[0] + 4) | ((mx[1] - mn[1] + 4) << 10) | ((mx[2] - mn[2] + 4) << 20));
}

__device__ __forceinline__ int ext_of(int packed, int a) { return (packed >> (10 * a)) & 1023; }

// Sums and maxima of one block's threads into info (one atomic per block).
__device__ __forceinline__ void info_add(unsigned long long* where, unsigned long long v) {
    __shared__ unsigned long long total;
    if (threadIdx.x == 0) total = 0;
    __syncthreads();
#pragma unroll
    for (int d = 16; d; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
    if ((threadIdx.x & 31) == 0 && v) atomicAdd(&total, v);
    __syncthreads();
    if (threadIdx.x == 0 && total) atomicAdd(where, total);
    __syncthreads();
}

// Element boxes of the three components (shared tables), box[c * elements +
// first + e]; the connectivity's (node, slot) pairs; info: site counts per
// component and a flag for anything the row form does not take (a node id or a
// box outside its range): the caller then uses the hash form, which reports it.
__global__ void __launch_bounds__(256) rows_boxes_kernel(const int64_t* __restrict__ base, int64_t total,
                                                         int64_t offset, const int64_t* __restrict__ cells, int group,
                                                         int64_t nq, int64_t first, int64_t elements, int64_t nodes,
                                                         FaceDims g, int4* __restrict__ box,
                                                         uint32_t* __restrict__ keys, int32_t* __restrict__ slots,
                                                         unsigned long long* info) {
    const int64_t e = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    unsigned long long sites[3] = {0, 0, 0};
    if (e < group) {
        bool ok = true;
        int64_t mn[2][3], mx[2][3];
#pragma unroll
        for (int l = 0; l < 2; ++l)
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                mn[l][a] = INT64_MAX;
                mx[l][a] = INT64_MIN;
            }
        for (int64_t q = 0; q < nq; ++q) {
            const int64_t row = offset + e * nq + q;
#pragma unroll
            for (int l = 0; l < 2; ++l)
#pragma unroll
                for (int a = 0; a < 3; ++a) {
                    const int64_t b = base[(int64_t(l) * total + row) * 3 + a];
                    mn[l][a] = b < mn[l][a] ? b : mn[l][a];
                    mx[l][a] = b > mx[l][a] ? b : mx[l][a];
                }
        }
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            int lo[3] = {0, 0, 0}, hi[3] = {0, 0, 0};
            unsigned long long n = 1;
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                const int l = a != c;
                const bool in = mn[l][a] >= 0 && support_inside(mx[l][a], face_n(g, c, a)) &&
                                mx[l][a] - mn[l][a] + 4 <= kMaxExt;
                ok = ok && in;
                lo[a] = in ? int(mn[l][a]) : 0;
                hi[a] = in ? int(mx[l][a]) : 0;
                n *= static_cast<unsigned long long>(hi[a] - lo[a] + 4);
            }
            box[c * elements + first + e] = pack_box(lo, hi);
            sites[c] = n;
        }
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            const int64_t node = cells[e * 4 + a];
            const bool in = node >= 0 && node < nodes;
            ok = ok && in;
            keys[(first + e) * 4 + a] = in ? uint32_t(node) : 0u;
            slots[(first + e) * 4 + a] = int32_t((first + e) * 4 + a);
        }
        if (!ok) atomicOr(info + AFSI_ROWS_FLAGS, 1ull);
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) info_add(info + AFSI_ROWS_SITES + c, sites[c]);
}

// start[k] = first position of key >= k in the sorted keys, k = 0..n_keys (a
// binary search per key; the keys are node ids, nearly all present).
__global__ void __launch_bounds__(256) rows_starts_kernel(const uint32_t* __restrict__ keys, int n, int n_keys,
                                                          int32_t* __restrict__ start) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k > n_keys) return;
    int lo = 0, hi = n;
    while (lo < hi) {
        const int mid = lo + ((hi - lo) >> 1);
        if (__ldg(keys + mid) < uint32_t(k))
            lo = mid + 1;
        else
            hi = mid;
    }
    start[k] = lo;
}

// Union box and volume of every node's cells (thread per component and node);
// info: padded entries per component, largest shared-memory box.
__global__ void __launch_bounds__(256) rows_node_boxes_kernel(const int4* __restrict__ box, int64_t elements,
                                                              const int32_t* __restrict__ start,
                                                              const int32_t* __restrict__ slots, int nodes,
                                                              int4* __restrict__ node_box, int64_t* __restrict__ volume,
                                                              unsigned long long* info) {
    const int n = blockIdx.x * blockDim.x + threadIdx.x, c = blockIdx.y;
    unsigned long long vol = 0, padded = 0;
    if (n < nodes) {
        int mn[3] = {INT_MAX, INT_MAX, INT_MAX}, mx[3] = {INT_MIN, INT_MIN, INT_MIN};
        const int s1 = start[n + 1];
        for (int k = start[n]; k < s1; ++k) {
            const int4 b = box[c * elements + (slots[k] >> 2)];
            const int lo[3] = {b.x, b.y, b.z};
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                mn[a] = min(mn[a], lo[a]);
                mx[a] = max(mx[a], lo[a] + ext_of(b.w, a) - 4);
            }
        }
        int4 nb = make_int4(0, 0, 0, 0);
        if (mx[0] >= mn[0]) {
            const bool fits = mx[0] - mn[0] + 4 <= kMaxExt && mx[1] - mn[1] + 4 <= kMaxExt && mx[2] - mn[2] + 4 <= kMaxExt;
            if (!fits) {
                atomicOr(info + AFSI_ROWS_FLAGS, 1ull);
            } else {
                nb = pack_box(mn, mx);
                int sx, sy;
                padded_strides(ext_of(nb.w, 1), ext_of(nb.w, 2), sx, sy);
                vol = static_cast<unsigned long long>(ext_of(nb.w, 0)) * ext_of(nb.w, 1) * ext_of(nb.w, 2);
                padded = static_cast<unsigned long long>(ext_of(nb.w, 0)) * sx;
            }
        }
        node_box[int64_t(c) * nodes + n] = nb;
        volume[int64_t(c) * nodes + n] = int64_t(vol);
    }
    info_add(info + AFSI_ROWS_PADDED + c, vol);
#pragma unroll
    for (int d = 16; d; d >>= 1) {
        const unsigned long long o = __shfl_xor_sync(0xffffffffu, padded, d);
        padded = o > padded ? o : padded;
    }
    if ((threadIdx.x & 31) == 0 && padded) atomicMax(info + AFSI_ROWS_BOX, padded);
}

template <class T>
struct RowGroups {
    int64_t offset[kRowsGroups];  // first table row
    const T* N[kRowsGroups];
    const T* W[kRowsGroups];
    int first[kRowsGroups];       // first element
    int nq[kRowsGroups];
    int count;
};

// Staged points and the cells they come from, per warp; the box follows.
template <class T>
struct __align__(16) RowsStage {
    T w[33 * 12];      // weight rows: x, y, z, four each; the last stays zero
    T f[33];           // W N[q,a]; the last stays zero
    int at[32];        // FP64: run key of the support origin in the box, FP32: its offset
    int perm[128], rs[33], rk[32];  // FP64: runs of one origin
    int pre[33];       // first point of each of the 32 current cells
    int grp[32];
    int64_t e4a[32];   // (element within its group) * 4 + a
};

template <class T> struct Neg0;
template <> struct Neg0<double> {
    static __device__ __forceinline__ bool is(double v) { return __double_as_longlong(v) == (long long)0x8000000000000000ull; }
};
template <> struct Neg0<float> {
    static __device__ __forceinline__ bool is(float v) { return __float_as_uint(v) == 0x80000000u; }
};

// Rows of B: one warp per (component, node), 4 warps per block.  `cap` is the
// largest padded box of any row (entries of dynamic shared memory per warp).
// FP32: lane (half, i, j) owns the link column (i, j) and z links 2 half,
// 2 half + 1 of each point; the padded strides keep a half-warp's 16 columns in distinct
// banks, and the links of one point are distinct entries, so the adds are
// plain read-modify-writes in point order.
template <class T>
__global__ void __launch_bounds__(kRowsWarps * 32) rows_fill_kernel(
    const int64_t* __restrict__ base, const T* __restrict__ phi, int64_t total,
    const __grid_constant__ RowGroups<T> groups,
    const int32_t* __restrict__ start, const int32_t* __restrict__ slots, int nodes, const int4* __restrict__ node_box,
    const int64_t* __restrict__ row_off, FaceDims g, int cap, int32_t* __restrict__ pcol, T* __restrict__ pval,
    int64_t* __restrict__ counts, unsigned long long* info) {
    extern __shared__ __align__(16) unsigned char rows_smem[];
    const size_t per = sizeof(RowsStage<T>) + (size_t(cap) * sizeof(T) + 15) / 16 * 16;
    RowsStage<T>& s = *reinterpret_cast<RowsStage<T>*>(rows_smem + (threadIdx.x >> 5) * per);
    T* acc = reinterpret_cast<T*>(reinterpret_cast<unsigned char*>(&s) + sizeof(RowsStage<T>));
    const int lane = threadIdx.x & 31, half = lane >> 4, li = (lane >> 2) & 3, lj = lane & 3;
    const int c = blockIdx.y;
    const int64_t warps = int64_t(gridDim.x) * kRowsWarps;
    constexpr bool mma = sizeof(T) == 8;
    if (lane < 12) s.w[32 * 12 + lane] = T(0);
    if (lane == 0) s.f[32] = T(0);
    using P = typename std::conditional<sizeof(T) == 8, double2, float2>::type;
    for (int64_t n = int64_t(blockIdx.x) * kRowsWarps + (threadIdx.x >> 5); n < nodes; n += warps) {
        const int4 nb = node_box[int64_t(c) * nodes + n];
        const int ex = ext_of(nb.w, 0), ey = ext_of(nb.w, 1), ez = ext_of(nb.w, 2);
        if (ex == 0) {
            if (lane == 0) counts[int64_t(c) * nodes + n] = 0;
            continue;
        }
        int sx, sy;
        padded_strides(ey, ez, sx, sy);
        __syncwarp();
        for (int t = lane; t < ex * sx; t += 32) acc[t] = -T(0);
        T* const mine = acc + li * sx + lj * sy + 2 * half;
        const int k1 = start[n + 1];
        for (int k0 = start[n]; k0 < k1; k0 += 32) {
            // the next 32 cells of the node: group, element, first point
            int nq = 0, grp = 0;
            int64_t e4a = 0;
            if (k0 + lane < k1) {
                const int slot = slots[k0 + lane], e = slot >> 2;
                while (grp + 1 < groups.count && e >= groups.first[grp + 1]) ++grp;
                nq = groups.nq[grp];
                e4a = int64_t(e - groups.first[grp]) * 4 + (slot & 3);
            }
            int pre = nq;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const int o = __shfl_up_sync(0xffffffffu, pre, d);
                if (lane >= d) pre += o;
            }
            const int points = __shfl_sync(0xffffffffu, pre, 31);
            __syncwarp();
            s.pre[lane + 1] = pre;
            if (lane == 0) s.pre[0] = 0;
            s.grp[lane] = grp;
            s.e4a[lane] = e4a;
            __syncwarp();
            for (int p0 = 0; p0 < points; p0 += 32) {
                const int m = min(32, points - p0), p = p0 + lane;
                T row[12], f = T(0);
                int at = 0;
                if (lane < m) {
                    int cell = 0;  // last cell with pre <= p
#pragma unroll
                    for (int d = 16; d; d >>= 1)
                        if (s.pre[cell + d] <= p) cell += d;
                    const int gi = s.grp[cell], q = p - s.pre[cell];
                    const int64_t ea = s.e4a[cell], local = (ea >> 2) * groups.nq[gi] + q;
                    const int64_t r0 = groups.offset[gi] + local;
                    f = groups.W[gi][local] * groups.N[gi][int64_t(q) * 4 + (ea & 3)];
                    const int lo[3] = {nb.x, nb.y, nb.z}, st[3] = {sx, sy, 1};
#pragma unroll
                    for (int a = 0; a < 3; ++a) {
                        const int64_t r = (int64_t(a != c) * total + r0) * 3 + a;
                        at += mma ? (int(base[r]) - lo[a]) << (10 * a) : (int(base[r]) - lo[a]) * st[a];
                        const P w0 = reinterpret_cast<const P*>(phi + r * 4)[0], w1 = reinterpret_cast<const P*>(phi + r * 4)[1];
                        row[a * 4] = w0.x;
                        row[a * 4 + 1] = w0.y;
                        row[a * 4 + 2] = w1.x;
                        row[a * 4 + 3] = w1.y;
                    }
                }
                __syncwarp();  // the previous points are done with the stage
                if (lane < m) {
                    P* dst = reinterpret_cast<P*>(s.w + lane * 12);
#pragma unroll
                    for (int k = 0; k < 6; ++k) {
                        P v;
                        v.x = row[2 * k];
                        v.y = row[2 * k + 1];
                        dst[k] = v;
                    }
                    s.f[lane] = f;
                    s.at[lane] = at;
                }
                __syncwarp();
                if constexpr (mma) {
                    spread_runs_mma<32, true>(acc, s.at, s.f, s.w, s.w + 4, s.w + 8, m, sx, sy, s.perm, s.rs, s.rk);
                } else for (int j = 0; j < m; ++j) {
                    const T* w = s.w + j * 12;
                    const T a = (w[li] * w[4 + lj]) * s.f[j];
                    const P z = *reinterpret_cast<const P*>(w + 8 + 2 * half);
                    T* dst = mine + s.at[j];
                    const T v0 = a * z.x, v1 = a * z.y;
                    if (v0 != T(0)) dst[0] += v0;
                    if (v1 != T(0)) dst[1] += v1;
                    __syncwarp();
                }
            }
        }
        // touched entries in ascending face order
        const int n1 = face_n(g, c, 1), n2 = face_n(g, c, 2);
        const int64_t off = row_off[int64_t(c) * nodes + n];
        const int cells = ex * ey * ez, qz = 32 % ez, q = 32 / ez, qy = q % ey, qx = q / ey;
        int z = lane % ez, r = lane / ez, y = r % ey, x = r / ey, written = 0;
        bool bad = false;
        for (int t0 = 0; t0 < cells; t0 += 32) {
            const bool in = t0 + lane < cells;
            const T v = in ? acc[x * sx + y * sy + z] : -T(0);
            const bool have = in && !Neg0<T>::is(v);
            const unsigned ballot = __ballot_sync(0xffffffffu, have);
            if (have) {
                const int64_t at = off + written + __popc(ballot & ((1u << lane) - 1u));
                pcol[at] = ((nb.x + x) * n1 + (nb.y + y)) * n2 + (nb.z + z);
                pval[at] = v;
                bad = bad || !isfinite(v);
            }
            written += __popc(ballot);
            z += qz;
            int carry = z >= ez ? 1 : 0;
            z -= carry * ez;
            y += qy + carry;
            carry = y >= ey ? 1 : 0;
            y -= carry * ey;
            x += qx + carry;
        }
        if (lane == 0) counts[int64_t(c) * nodes + n] = written;
        if (bad) atomicOr(info + AFSI_ROWS_FLAGS, 2ull);
    }
}

// Padded rows to CSR, with the sort input of the transpose (face, position)
// and the row of every entry.  One warp per row.
template <class T>
__global__ void __launch_bounds__(256) rows_pack_kernel(const int64_t* __restrict__ crow, const int64_t* __restrict__ row_off,
                                                        int nodes, const int32_t* __restrict__ pcol,
                                                        const T* __restrict__ pval, int64_t* __restrict__ col,
                                                        T* __restrict__ val, uint32_t* __restrict__ key,
                                                        int32_t* __restrict__ pos, int32_t* __restrict__ row) {
    const int64_t n = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    if (n >= nodes) return;
    const int64_t a = crow[n], b = crow[n + 1], off = row_off[n] - a;
    for (int64_t i = a + (threadIdx.x & 31); i < b; i += 32) {
        const int32_t f = pcol[off + i];
        col[i] = f;
        val[i] = pval[off + i];
        key[i] = uint32_t(f);
        pos[i] = int32_t(i);
        row[i] = int32_t(n);
    }
}

// Entries of the transpose in sorted order; run lengths of the keys into count
// (zeroed): -first at a run's first entry, last + 1 at its last.
template <class T>
__global__ void __launch_bounds__(256) rows_transpose_kernel(const uint32_t* __restrict__ key,
                                                             const int32_t* __restrict__ pos, int64_t n,
                                                             const T* __restrict__ val, const int32_t* __restrict__ row,
                                                             int64_t* __restrict__ t_col, T* __restrict__ t_val,
                                                             unsigned long long* __restrict__ count) {
    for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x) {
        const int32_t p = pos[i];
        t_val[i] = val[p];
        t_col[i] = row[p];
        const uint32_t k = key[i];
        if (i == 0 || key[i - 1] != k) atomicAdd(count + k, 0ull - static_cast<unsigned long long>(i));
        if (i + 1 == n || key[i + 1] != k) atomicAdd(count + k, static_cast<unsigned long long>(i) + 1ull);
    }
}

inline int64_t slab(int64_t bytes) { return (bytes + 255) / 256 * 256; }

inline int bits_for(int64_t limit) {  // bits that hold 0..limit-1
    int b = 1;
    while (b < 32 && (int64_t(1) << b) < limit) ++b;
    return b;
}

size_t pair_sort_bytes(int64_t n, int bits) {
    size_t t = 0;
    cub::DeviceRadixSort::SortPairs(nullptr, t, static_cast<const uint32_t*>(nullptr), static_cast<uint32_t*>(nullptr),
                                    static_cast<const int32_t*>(nullptr), static_cast<int32_t*>(nullptr), n, 0, bits);
    return t;
}

size_t scan_bytes(int64_t n) {
    size_t t = 0;
    cub::DeviceScan::ExclusiveSum(nullptr, t, static_cast<const int64_t*>(nullptr), static_cast<int64_t*>(nullptr), n);
    return t;
}

int32_t check_rows(int64_t elements, int64_t nodes, int64_t nx, int64_t ny, int64_t nz) {
    AFSI_REQUIRE(elements > 0 && elements <= INT32_MAX / 4 && nodes > 0 && nodes < INT32_MAX, "invalid row assembly sizes");
    AFSI_REQUIRE(nx > 0 && ny > 0 && nz > 0 && nx < (1 << 20) && ny < (1 << 20) && nz < (1 << 20) &&
                     (nx + 1) * (ny + 1) * (nz + 1) < INT32_MAX,
                 "face arrays too large for the row assembly");
    return AFSI_OK;
}

template <class T>
size_t fill_smem(int64_t cap) {
    return kRowsWarps * (sizeof(RowsStage<T>) + (size_t(cap) * sizeof(T) + 15) / 16 * 16);
}

constexpr size_t kRowsSmem = 200 * 1024;

}  // namespace
}  // namespace afsi

using namespace afsi;

extern "C" int64_t afsi_b200_p1_rows_cap(int32_t dtype) {
    const int64_t room = int64_t(kRowsSmem) / kRowsWarps;
    return dtype == AFSI_F64 ? (room - int64_t(sizeof(RowsStage<double>))) / 8 - 2
                             : (room - int64_t(sizeof(RowsStage<float>))) / 4 - 4;
}

extern "C" int64_t afsi_b200_p1_rows_scratch_bytes(int64_t elements, int64_t nodes, int64_t nnz, int64_t nf) {
    if (elements < 0 || nodes < 0 || nnz < 0 || nf < 0) return -1;
    const size_t plan = std::max(pair_sort_bytes(std::max<int64_t>(4 * elements, 1), 32),
                                 scan_bytes(std::max<int64_t>(3 * nodes, 1)));
    const size_t fin = std::max(pair_sort_bytes(std::max<int64_t>(nnz, 1), 32), scan_bytes(nf + 1));
    return std::max<int64_t>(slab(elements * 16) + slab(int64_t(plan)), 5 * slab(nnz * 4) + slab(int64_t(fin)));
}

extern "C" int32_t afsi_b200_p1_rows_boxes(const int64_t* base, int64_t total, int64_t offset, const int64_t* cells,
                                           int64_t group_elements, int64_t nq, int64_t first, int64_t elements,
                                           int64_t nodes, int64_t nx, int64_t ny, int64_t nz, int32_t* box,
                                           uint32_t* keys, int32_t* slots, uint64_t* info, afsi_stream_t stream) {
    int32_t rc = check_rows(elements, nodes, nx, ny, nz);
    if (rc) return rc;
    AFSI_REQUIRE(group_elements >= 0 && nq > 0 && first >= 0 && first + group_elements <= elements,
                 "invalid IB group sizes");
    AFSI_REQUIRE(offset >= 0 && offset <= total && group_elements * nq <= total - offset, "IB group offset is out of range");
    if (group_elements == 0) return AFSI_OK;
    AFSI_REQUIRE(base && cells && box && keys && slots && info, "null device pointer");
    rows_boxes_kernel<<<blocks_for(group_elements, 256), 256, 0, stream>>>(
        base, total, offset, cells, int(group_elements), nq, first, elements, nodes,
        FaceDims{int(nx), int(ny), int(nz)}, reinterpret_cast<int4*>(box), keys, slots,
        reinterpret_cast<unsigned long long*>(info));
    return launched("p1_rows_boxes");
}

extern "C" int32_t afsi_b200_p1_rows_incidence(const int32_t* box, int64_t elements, int64_t nodes,
                                               const uint32_t* keys, const int32_t* slots_in, int32_t* start,
                                               int32_t* slots, int32_t* node_box, int64_t* volume, int64_t* row_off,
                                               uint64_t* info, void* scratch, int64_t scratch_bytes,
                                               afsi_stream_t stream) {
    int32_t rc = check_rows(elements, nodes, 1, 1, 1);
    if (rc) return rc;
    AFSI_REQUIRE(box && keys && slots_in && start && slots && node_box && volume && row_off && info && scratch,
                 "null device pointer");
    AFSI_REQUIRE(scratch_bytes >= afsi_b200_p1_rows_scratch_bytes(elements, nodes, 0, 0), "row assembly scratch too small");
    uint32_t* sorted = static_cast<uint32_t*>(scratch);
    unsigned char* temp = static_cast<unsigned char*>(scratch) + slab(elements * 16);
    size_t temp_bytes = size_t(scratch_bytes - slab(elements * 16));
    if (cub::DeviceRadixSort::SortPairs(temp, temp_bytes, keys, sorted, slots_in, slots, elements * 4, 0,
                                        bits_for(nodes), stream) != cudaSuccess)
        return fail(AFSI_ERR_CUDA, "connectivity sort failed");
    rows_starts_kernel<<<blocks_for(nodes + 1, 256), 256, 0, stream>>>(sorted, int(elements * 4), int(nodes), start);
    rows_node_boxes_kernel<<<dim3(blocks_for(nodes, 256), 3), 256, 0, stream>>>(
        reinterpret_cast<const int4*>(box), elements, start, slots, int(nodes), reinterpret_cast<int4*>(node_box),
        volume, reinterpret_cast<unsigned long long*>(info));
    if ((rc = launched("p1_rows_incidence"))) return rc;
    temp_bytes = size_t(scratch_bytes - slab(elements * 16));
    if (cub::DeviceScan::ExclusiveSum(temp, temp_bytes, volume, row_off, 3 * nodes, stream) != cudaSuccess)
        return fail(AFSI_ERR_CUDA, "row offset scan failed");
    return launched("p1_rows_incidence scan");
}

extern "C" int32_t afsi_b200_p1_rows_fill(const int64_t* base, const void* phi, int64_t total,
                                          const afsi_rows_group* groups, int32_t group_count, const int32_t* start,
                                          const int32_t* slots, int64_t nodes, const int32_t* node_box,
                                          const int64_t* row_off, int64_t nx, int64_t ny, int64_t nz, int64_t box_cap,
                                          int32_t* pcol, void* pval, int64_t* counts, uint64_t* info, int32_t dtype,
                                          afsi_stream_t stream) {
    int32_t rc = check_rows(1, nodes, nx, ny, nz);
    if (rc) return rc;
    AFSI_REQUIRE(groups && group_count >= 1 && group_count <= kRowsGroups, "1 to %d quadrature groups", kRowsGroups);
    AFSI_REQUIRE(base && phi && start && slots && node_box && row_off && pcol && pval && counts && info,
                 "null device pointer");
    AFSI_REQUIRE(reinterpret_cast<uintptr_t>(phi) % 16 == 0, "IB weight table must be 16-byte aligned");
    AFSI_REQUIRE(box_cap > 0 && box_cap <= afsi_b200_p1_rows_cap(dtype), "row box exceeds shared memory");
    AFSI_DISPATCH(dtype, {
        RowGroups<T> gr = {};
        gr.count = group_count;
        for (int k = 0; k < group_count; ++k) {
            AFSI_REQUIRE(groups[k].N && groups[k].W && groups[k].nq > 0 && groups[k].nq <= (1 << 20) &&
                             groups[k].first >= 0 && groups[k].first <= INT32_MAX / 4,
                         "invalid quadrature group");
            gr.offset[k] = groups[k].offset;
            gr.N[k] = static_cast<const T*>(groups[k].N);
            gr.W[k] = static_cast<const T*>(groups[k].W);
            gr.first[k] = int(groups[k].first);
            gr.nq[k] = int(groups[k].nq);
        }
        const size_t smem = fill_smem<T>(box_cap);
        if ((rc = allow_shared<rows_fill_kernel<T>>("p1_rows_fill", kRowsSmem + 4096))) return rc;
        const int64_t want = (nodes + kRowsWarps - 1) / kRowsWarps;
        rows_fill_kernel<T><<<dim3(unsigned(std::min<int64_t>(want, 1 << 20)), 3), kRowsWarps * 32, smem, stream>>>(
            base, static_cast<const T*>(phi), total, gr, start, slots, int(nodes),
            reinterpret_cast<const int4*>(node_box), row_off, FaceDims{int(nx), int(ny), int(nz)}, int(box_cap), pcol,
            static_cast<T*>(pval), counts, reinterpret_cast<unsigned long long*>(info));
    });
    return launched("p1_rows_fill");
}

extern "C" int32_t afsi_b200_p1_rows_pointers(const int64_t* counts, int64_t nodes, int64_t* crow, void* scratch,
                                              int64_t scratch_bytes, afsi_stream_t stream) {
    AFSI_REQUIRE(nodes > 0 && counts && crow && scratch, "invalid row pointer arguments");
    size_t temp = size_t(scratch_bytes);
    AFSI_REQUIRE(scan_bytes(nodes) <= temp, "row pointer scratch too small");
    if (cudaMemsetAsync(crow, 0, sizeof(int64_t), stream) != cudaSuccess)
        return fail(AFSI_ERR_CUDA, "row pointer clear failed");
    if (cub::DeviceScan::InclusiveSum(scratch, temp, counts, crow + 1, nodes, stream) != cudaSuccess)
        return fail(AFSI_ERR_CUDA, "row pointer scan failed");
    return launched("p1_rows_pointers");
}

extern "C" int32_t afsi_b200_p1_rows_finish(const int64_t* crow, const int64_t* row_off, int64_t nodes,
                                            const int32_t* pcol, const void* pval, int64_t nnz, int64_t nf,
                                            int64_t* col, void* val, int64_t* t_crow, int64_t* t_col, void* t_val,
                                            void* scratch, int64_t scratch_bytes, int32_t dtype, afsi_stream_t stream) {
    AFSI_REQUIRE(nodes > 0 && nodes < INT32_MAX && nf > 0 && nf < INT32_MAX && nnz >= 0 && nnz < INT32_MAX,
                 "invalid CSR sizes");
    AFSI_REQUIRE(crow && row_off && t_crow && scratch, "null device pointer");
    AFSI_REQUIRE(scratch_bytes >= afsi_b200_p1_rows_scratch_bytes(0, 0, nnz, nf), "row assembly scratch too small");
    if (cudaMemsetAsync(t_crow, 0, size_t(nf + 1) * 8, stream) != cudaSuccess)
        return fail(AFSI_ERR_CUDA, "transpose pointer clear failed");
    if (nnz == 0) return AFSI_OK;
    AFSI_REQUIRE(pcol && pval && col && val && t_col && t_val, "null device pointer");
    unsigned char* p = static_cast<unsigned char*>(scratch);
    const int64_t step = slab(nnz * 4);
    uint32_t* key = reinterpret_cast<uint32_t*>(p);
    uint32_t* key_sorted = reinterpret_cast<uint32_t*>(p + step);
    int32_t* pos = reinterpret_cast<int32_t*>(p + 2 * step);
    int32_t* pos_sorted = reinterpret_cast<int32_t*>(p + 3 * step);
    int32_t* row = reinterpret_cast<int32_t*>(p + 4 * step);
    void* temp = p + 5 * step;
    const size_t room = size_t(scratch_bytes - 5 * step);
    AFSI_DISPATCH(dtype, {
        rows_pack_kernel<T><<<blocks_for(nodes * 32, 256), 256, 0, stream>>>(
            crow, row_off, int(nodes), pcol, static_cast<const T*>(pval), col, static_cast<T*>(val), key, pos, row);
        int32_t rc = launched("p1_rows_pack");
        if (rc) return rc;
        size_t bytes = room;
        if (cub::DeviceRadixSort::SortPairs(temp, bytes, key, key_sorted, pos, pos_sorted, nnz, 0, bits_for(nf), stream) !=
            cudaSuccess)
            return fail(AFSI_ERR_CUDA, "CSR transpose sort failed");
        const unsigned grid = unsigned(std::min<int64_t>((nnz + 255) / 256, 148 * 16));
        rows_transpose_kernel<T><<<grid, 256, 0, stream>>>(key_sorted, pos_sorted, nnz, static_cast<const T*>(val), row,
                                                           t_col, static_cast<T*>(t_val),
                                                           reinterpret_cast<unsigned long long*>(t_crow));
        if ((rc = launched("p1_rows_transpose"))) return rc;
        bytes = room;
        if (cub::DeviceScan::ExclusiveSum(temp, bytes, t_crow, t_crow, nf + 1, stream) != cudaSuccess)
            return fail(AFSI_ERR_CUDA, "transpose pointer scan failed");
    });
    return launched("p1_rows_finish");
}
