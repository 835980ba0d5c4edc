// IB_4 spread / gather kernels: indexed (explicit ids) and compact separable
// 3D, plus the C-ABI of the fused P2 element transfers whose kernels live in
// p2.cu.
//
// Gather kernels are atomic-free and deterministic.  Spreads add into zeroed
// fields with fire-and-forget L2 reductions.
//
// What bounds the compact transfers is the number of 32-byte sectors that
// their field accesses touch in the L2: marker clouds have no order, so a
// point's 64 links are 16 rows of four consecutive values anywhere in the face
// array.  Each point is therefore a group of four lanes, lane k owning z link
// k: one instruction of a warp touches eight rows, whose four values fall into
// one or two sectors, where a lane per x offset touched 32 sectors.  All three
// components run in one launch (grid y), reading the force and writing the
// velocities in their (P, 3) layout.  400,000 markers on 64^3, FP64, one B200:
// spread 668 -> 305 us (110 G sector reductions/s, the L2's rate either way),
// gather 172 -> 81 us.  Clouds with many points per cell take the binned spread
// (compact_bins.cu).  The 2D pair (20,000 markers, 256 x 64) is bound by
// launches: 29 -> 8 us of spread and 12 device operations -> 7 for a transfer.
#include <cmath>
#include "common.cuh"
#include "p2.cuh"

namespace afsi {

// ----------------------------------------------------------------- indexed

// G lanes per (point, component); G = 16 for the 2D 4x4 stencils.
template <class T, bool Spread, int G>
__global__ void __launch_bounds__(256) indexed_kernel(const T* __restrict__ f, const int64_t* __restrict__ ids,
                                                      const T* __restrict__ w, T* __restrict__ out, int64_t points,
                                                      int64_t neighbors, int64_t components, int64_t nodes,
                                                      T volume, int32_t* status) {
    const int64_t task = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) / G;
    const int sub = threadIdx.x % G;
    const bool active = task < points * components;
    const int64_t p = active ? task / components : 0, c = active ? task % components : 0;
    T sum = T(0);
    if (active) {
        for (int64_t k = sub; k < neighbors; k += G) {
            const int64_t j = ids[p * neighbors + k];
            if (j < 0 || j >= nodes) {
                flag(status, AFSI_FLAG_INDEX);
                continue;
            }
            const T weight = w[p * neighbors + k];
            if (Spread)
                atomicAdd(out + j * components + c, (f[p * components + c] * weight) / volume);
            else
                sum += f[j * components + c] * weight;
        }
    }
    if (!Spread) {
#pragma unroll
        for (int d = G / 2; d; d >>= 1) sum += __shfl_down_sync(0xffffffffu, sum, d, G);
        if (active && sub == 0) out[p * components + c] = sum;
    }
}

// The two components of a 2D channel transfer in one launch (grid y), 16 taps
// per point: u, v arrays of one value per face, point data with `stride`
// values per point.
template <class T>
struct Pair2D {
    const int64_t* ids[2];
    const T* w[2];
    const T* in[2];
    T* out[2];
    int64_t nodes[2];
};

template <class T, bool Spread>
__global__ void __launch_bounds__(256) indexed_pair_kernel(Pair2D<T> a, int64_t points, int64_t stride, T volume,
                                                           T inv_volume, int32_t* status) {
    const int c = blockIdx.y;
    const int64_t p = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 4;
    const int sub = threadIdx.x & 15;
    const bool active = p < points;
    T sum = T(0);
    if (active) {
        const int64_t j = (c ? a.ids[1] : a.ids[0])[p * 16 + sub];
        const T weight = (c ? a.w[1] : a.w[0])[p * 16 + sub];
        if (j < 0 || j >= (c ? a.nodes[1] : a.nodes[0])) {
            flag(status, AFSI_FLAG_INDEX);
        } else if (Spread) {
            const T fw = (c ? a.in[1] : a.in[0])[p * stride] * weight;
            atomicAdd((c ? a.out[1] : a.out[0]) + j, inv_volume != T(0) ? fw * inv_volume : fw / volume);
        } else {
            sum = (c ? a.in[1] : a.in[0])[j] * weight;
        }
    }
    if (!Spread) {
#pragma unroll
        for (int d = 8; d; d >>= 1) sum += __shfl_down_sync(0xffffffffu, sum, d, 16);
        if (active && sub == 0) (c ? a.out[1] : a.out[0])[p * stride] = sum;
    }
}

// ----------------------------------------------------------------- compact

// False (and the caller flags) if the 4x4x4 box leaves [0,n).
__device__ __forceinline__ bool box_inside(int64_t bx, int64_t by, int64_t bz, int64_t nx, int64_t ny, int64_t nz) {
    return support_inside(bx, nx) && support_inside(by, ny) && support_inside(bz, nz);
}

// Components of one launch: face arrays and their dims, tables of the first
// component (the others follow at points * 3 and points * 12), point values
// with `stride` per point.
template <class T>
struct CompactArgs {
    T* field[3];
    int64_t n[3][3];
    const int64_t* base;
    const T* phi;
    int64_t points, stride;
    T* values;
};

template <class T> struct CompactVec;
template <> struct CompactVec<double> { using type = double2; };
template <> struct CompactVec<float> { using type = float4; };

// Four weights at w: as 16-byte loads when the table is aligned for them.
template <class T, bool Aligned>
__device__ __forceinline__ void load4(const T* __restrict__ w, T out[4]) {
    if constexpr (Aligned) {
        using V = typename CompactVec<T>::type;
        constexpr int per = 16 / int(sizeof(T));
#pragma unroll
        for (int k = 0; k < 4 / per; ++k) {
            const V v = reinterpret_cast<const V*>(w)[k];
            const T* e = reinterpret_cast<const T*>(&v);
#pragma unroll
            for (int i = 0; i < per; ++i) out[k * per + i] = e[i];
        }
    } else {
#pragma unroll
        for (int k = 0; k < 4; ++k) out[k] = w[k];
    }
}

template <class T, bool Spread, bool Aligned>
__global__ void __launch_bounds__(256) compact_kernel(CompactArgs<T> a, T volume, T inv_volume, int32_t* status) {
    const int c = blockIdx.y;
    const int64_t p = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 2;
    const int k = threadIdx.x & 3;
    const bool active = p < a.points;
    T* field = c == 0 ? a.field[0] : c == 1 ? a.field[1] : a.field[2];
    const int64_t nx = c == 0 ? a.n[0][0] : c == 1 ? a.n[1][0] : a.n[2][0];
    const int64_t ny = c == 0 ? a.n[0][1] : c == 1 ? a.n[1][1] : a.n[2][1];
    const int64_t nz = c == 0 ? a.n[0][2] : c == 1 ? a.n[1][2] : a.n[2][2];
    T sum = T(0);
    if (active) {
        const int64_t row = c * a.points + p;
        const int64_t bx = a.base[row * 3], by = a.base[row * 3 + 1], bz = a.base[row * 3 + 2];
        if (!box_inside(bx, by, bz, nx, ny, nz)) {
            if (k == 0) flag(status, AFSI_FLAG_INDEX);
        } else {
            const T* ph = a.phi + row * 12;
            T px[4], py[4];
            load4<T, Aligned>(ph, px);
            load4<T, Aligned>(ph + 4, py);
            const T pz = ph[8 + k];
            T* at = field + (bx * ny + by) * nz + bz + k;
            const int64_t sx = ny * nz;
            if (Spread) {
                const T fv = a.values[p * a.stride + c];
                const T fz = (inv_volume != T(0) ? fv * inv_volume : fv / volume) * pz;
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) atomicAdd(at + i * sx + j * nz, (px[i] * py[j]) * fz);
            } else {
                T v[4][4];
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) v[i][j] = at[i * sx + j * nz];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    T r = v[i][0] * py[0];
#pragma unroll
                    for (int j = 1; j < 4; ++j) r = fma(v[i][j], py[j], r);
                    sum = fma(r, px[i], sum);
                }
                sum *= pz;
            }
        }
    }
    if (!Spread) {
        sum += __shfl_xor_sync(0xffffffffu, sum, 1);
        sum += __shfl_xor_sync(0xffffffffu, sum, 2);
        if (active && k == 0) a.values[p * a.stride + c] = sum;
    }
}

// rhs[n] (+)= sum over the node's (element, slot) entries in CSR order.
template <class T>
__global__ void __launch_bounds__(256) node_reduce_kernel(const T* __restrict__ local, int64_t slots,
                                                          const int64_t* __restrict__ crow,
                                                          const int64_t* __restrict__ slot, int64_t nodes,
                                                          T* __restrict__ rhs, int accumulate, int32_t* status) {
    const int64_t n = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (n >= nodes) return;
    T s[3] = {T(0), T(0), T(0)};
    for (int64_t k = crow[n]; k < crow[n + 1]; ++k) {
        const int64_t s_ = slot[k];
        if (s_ < 0 || s_ >= slots) {
            flag(status, AFSI_FLAG_INDEX);
            continue;
        }
#pragma unroll
        for (int c = 0; c < 3; ++c) s[c] += local[s_ * 3 + c];
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) rhs[n * 3 + c] = accumulate ? rhs[n * 3 + c] + s[c] : s[c];
}

}  // namespace afsi

using namespace afsi;

extern "C" int32_t afsi_b200_indexed_gather(const void* field, int64_t nodes, int64_t components,
                                            const int64_t* ids, const void* weights, int64_t points,
                                            int64_t neighbors, void* out, int32_t* status, int32_t dtype,
                                            afsi_stream_t stream) {
    AFSI_REQUIRE(nodes > 0 && components > 0 && neighbors > 0 && points >= 0, "invalid indexed gather sizes");
    if (points == 0) return AFSI_OK;
    AFSI_REQUIRE(field && ids && weights && out, "null device pointer");
    const int64_t tasks = points * components;
    AFSI_DISPATCH(dtype, {
        if (neighbors <= 16)
            indexed_kernel<T, false, 16><<<blocks_for(tasks * 16, 256), 256, 0, stream>>>(
                static_cast<const T*>(field), ids, static_cast<const T*>(weights), static_cast<T*>(out), points,
                neighbors, components, nodes, T(1), status);
        else
            indexed_kernel<T, false, 32><<<blocks_for(tasks * 32, 256), 256, 0, stream>>>(
                static_cast<const T*>(field), ids, static_cast<const T*>(weights), static_cast<T*>(out), points,
                neighbors, components, nodes, T(1), status);
    });
    return launched("indexed_gather");
}

extern "C" int32_t afsi_b200_indexed_spread(const void* field, int64_t points, int64_t components,
                                            const int64_t* ids, const void* weights, int64_t neighbors,
                                            int64_t size, double volume, void* out, int32_t* status, int32_t dtype,
                                            afsi_stream_t stream) {
    AFSI_REQUIRE(size > 0 && components > 0 && neighbors > 0 && points >= 0, "invalid indexed spread sizes");
    AFSI_REQUIRE(isfinite(volume) && volume > 0, "invalid IB output size/volume");
    if (points == 0) return AFSI_OK;
    AFSI_REQUIRE(field && ids && weights && out, "null device pointer");
    const int64_t tasks = points * components;
    AFSI_DISPATCH(dtype, {
        if (neighbors <= 16)
            indexed_kernel<T, true, 16><<<blocks_for(tasks * 16, 256), 256, 0, stream>>>(
                static_cast<const T*>(field), ids, static_cast<const T*>(weights), static_cast<T*>(out), points,
                neighbors, components, size, T(volume), status);
        else
            indexed_kernel<T, true, 32><<<blocks_for(tasks * 32, 256), 256, 0, stream>>>(
                static_cast<const T*>(field), ids, static_cast<const T*>(weights), static_cast<T*>(out), points,
                neighbors, components, size, T(volume), status);
    });
    return launched("indexed_spread");
}

namespace {

template <class T, bool Spread>
int32_t launch_compact(const CompactArgs<T>& a, int components, double volume, int32_t* status, cudaStream_t stream) {
    const dim3 grid(blocks_for(a.points * 4, 256), unsigned(components));
    const T vol = T(volume), inv = Spread ? exact_inverse(vol) : T(0);
    // a component's table starts points * 12 values after the previous one's
    const bool aligned = reinterpret_cast<uintptr_t>(a.phi) % 16 == 0;
    if (aligned)
        compact_kernel<T, Spread, true><<<grid, 256, 0, stream>>>(a, vol, inv, status);
    else
        compact_kernel<T, Spread, false><<<grid, 256, 0, stream>>>(a, vol, inv, status);
    return launched(Spread ? "compact_spread" : "compact_gather");
}

// One component: its own array, tables and contiguous values.
template <class T>
CompactArgs<T> one_component(const void* field, const int64_t* base, const void* phi, int64_t points, int64_t nx,
                             int64_t ny, int64_t nz, const void* values) {
    CompactArgs<T> a = {};
    a.field[0] = const_cast<T*>(static_cast<const T*>(field));
    a.n[0][0] = nx;
    a.n[0][1] = ny;
    a.n[0][2] = nz;
    a.base = base;
    a.phi = static_cast<const T*>(phi);
    a.points = points;
    a.stride = 1;
    a.values = const_cast<T*>(static_cast<const T*>(values));
    return a;
}

// The three face arrays of an (nx, ny, nz) cell grid, point values (points, 3).
template <class T>
CompactArgs<T> three_components(const void* u0, const void* u1, const void* u2, const int64_t* base, const void* phi,
                                int64_t points, int64_t nx, int64_t ny, int64_t nz, const void* values) {
    CompactArgs<T> a = one_component<T>(u0, base, phi, points, nx, ny, nz, values);
    a.field[1] = const_cast<T*>(static_cast<const T*>(u1));
    a.field[2] = const_cast<T*>(static_cast<const T*>(u2));
    for (int c = 0; c < 3; ++c) {
        a.n[c][0] = nx + (c == 0);
        a.n[c][1] = ny + (c == 1);
        a.n[c][2] = nz + (c == 2);
    }
    a.stride = 3;
    return a;
}

}  // namespace

extern "C" int32_t afsi_b200_compact_gather(const void* field, const int64_t* base, const void* phi,
                                            int64_t points, int64_t nx, int64_t ny, int64_t nz, void* out,
                                            int32_t* status, int32_t dtype, afsi_stream_t stream) {
    AFSI_REQUIRE(nx > 0 && ny > 0 && nz > 0 && points >= 0, "invalid compact grid");
    if (points == 0) return AFSI_OK;
    AFSI_REQUIRE(field && base && phi && out, "null device pointer");
    AFSI_DISPATCH(dtype, {
        return launch_compact<T, false>(one_component<T>(field, base, phi, points, nx, ny, nz, out), 1, 1.0, status,
                                        stream);
    });
    return AFSI_OK;
}

extern "C" int32_t afsi_b200_compact_spread(const void* field, const int64_t* base, const void* phi,
                                            int64_t points, int64_t nx, int64_t ny, int64_t nz, double volume,
                                            void* out, int32_t* status, int32_t dtype, afsi_stream_t stream) {
    AFSI_REQUIRE(nx > 0 && ny > 0 && nz > 0 && points >= 0, "invalid compact grid");
    AFSI_REQUIRE(isfinite(volume) && volume > 0, "invalid compact grid/volume");
    if (points == 0) return AFSI_OK;
    AFSI_REQUIRE(field && base && phi && out, "null device pointer");
    AFSI_DISPATCH(dtype, {
        return launch_compact<T, true>(one_component<T>(out, base, phi, points, nx, ny, nz, field), 1, volume, status,
                                       stream);
    });
    return AFSI_OK;
}

extern "C" int32_t afsi_b200_compact_gather3(const void* u0, const void* u1, const void* u2, const int64_t* base,
                                             const void* phi, int64_t points, int64_t nx, int64_t ny, int64_t nz,
                                             void* out, int32_t* status, int32_t dtype, afsi_stream_t stream) {
    AFSI_REQUIRE(nx > 0 && ny > 0 && nz > 0 && points >= 0, "invalid compact grid");
    if (points == 0) return AFSI_OK;
    AFSI_REQUIRE(u0 && u1 && u2 && base && phi && out, "null device pointer");
    AFSI_DISPATCH(dtype, {
        return launch_compact<T, false>(three_components<T>(u0, u1, u2, base, phi, points, nx, ny, nz, out), 3, 1.0,
                                        status, stream);
    });
    return AFSI_OK;
}

extern "C" int32_t afsi_b200_compact_spread3(const void* force, const int64_t* base, const void* phi, int64_t points,
                                             int64_t nx, int64_t ny, int64_t nz, double volume, void* u0, void* u1,
                                             void* u2, int32_t* status, int32_t dtype, afsi_stream_t stream) {
    AFSI_REQUIRE(nx > 0 && ny > 0 && nz > 0 && points >= 0, "invalid compact grid");
    AFSI_REQUIRE(isfinite(volume) && volume > 0, "invalid compact grid/volume");
    AFSI_REQUIRE(u0 && u1 && u2, "null device pointer");
    const size_t es = dtype == AFSI_F64 ? 8 : 4;
    if (cudaMemsetAsync(u0, 0, size_t((nx + 1) * ny * nz) * es, stream) != cudaSuccess ||
        cudaMemsetAsync(u1, 0, size_t(nx * (ny + 1) * nz) * es, stream) != cudaSuccess ||
        cudaMemsetAsync(u2, 0, size_t(nx * ny * (nz + 1)) * es, stream) != cudaSuccess)
        return fail(AFSI_ERR_CUDA, "clearing the face arrays failed");
    if (points == 0) return AFSI_OK;
    AFSI_REQUIRE(force && base && phi, "null device pointer");
    AFSI_DISPATCH(dtype, {
        return launch_compact<T, true>(three_components<T>(u0, u1, u2, base, phi, points, nx, ny, nz, force), 3, volume,
                                       status, stream);
    });
    return AFSI_OK;
}

extern "C" int32_t afsi_b200_indexed_gather2(const void* u, const void* v, int64_t nu, int64_t nv, const int64_t* ids0,
                                             const int64_t* ids1, const void* w0, const void* w1, int64_t points,
                                             void* out, int32_t* status, int32_t dtype, afsi_stream_t stream) {
    AFSI_REQUIRE(nu > 0 && nv > 0 && points >= 0, "invalid indexed gather sizes");
    if (points == 0) return AFSI_OK;
    AFSI_REQUIRE(u && v && ids0 && ids1 && w0 && w1 && out, "null device pointer");
    AFSI_DISPATCH(dtype, {
        const Pair2D<T> a{{ids0, ids1},
                          {static_cast<const T*>(w0), static_cast<const T*>(w1)},
                          {static_cast<const T*>(u), static_cast<const T*>(v)},
                          {static_cast<T*>(out), static_cast<T*>(out) + 1},
                          {nu, nv}};
        indexed_pair_kernel<T, false><<<dim3(blocks_for(points * 16, 256), 2), 256, 0, stream>>>(a, points, 2, T(1), T(0),
                                                                                               status);
    });
    return launched("indexed_gather2");
}

extern "C" int32_t afsi_b200_indexed_spread2(const void* force, int64_t stride, const int64_t* ids0,
                                             const int64_t* ids1, const void* w0, const void* w1, int64_t points,
                                             int64_t nu, int64_t nv, double volume, void* u, void* v, int32_t* status,
                                             int32_t dtype, afsi_stream_t stream) {
    AFSI_REQUIRE(nu > 0 && nv > 0 && points >= 0 && stride >= 2, "invalid indexed spread sizes");
    AFSI_REQUIRE(isfinite(volume) && volume > 0, "invalid IB output size/volume");
    AFSI_REQUIRE(u && v, "null device pointer");
    const size_t es = dtype == AFSI_F64 ? 8 : 4;
    if (cudaMemsetAsync(u, 0, size_t(nu) * es, stream) != cudaSuccess ||
        cudaMemsetAsync(v, 0, size_t(nv) * es, stream) != cudaSuccess)
        return fail(AFSI_ERR_CUDA, "clearing the face arrays failed");
    if (points == 0) return AFSI_OK;
    AFSI_REQUIRE(force && ids0 && ids1 && w0 && w1, "null device pointer");
    AFSI_DISPATCH(dtype, {
        const Pair2D<T> a{{ids0, ids1},
                          {static_cast<const T*>(w0), static_cast<const T*>(w1)},
                          {static_cast<const T*>(force), static_cast<const T*>(force) + 1},
                          {static_cast<T*>(u), static_cast<T*>(v)},
                          {nu, nv}};
        indexed_pair_kernel<T, true><<<dim3(blocks_for(points * 16, 256), 2), 256, 0, stream>>>(
            a, points, stride, T(volume), exact_inverse(T(volume)), status);
    });
    return launched("indexed_spread2");
}

static int32_t p2_check(int64_t elements, int64_t nq, int64_t total, int64_t offset, int64_t nx, int64_t ny,
                        int64_t nz) {
    AFSI_REQUIRE(elements >= 0 && nq > 0, "invalid P2 group sizes");
    AFSI_REQUIRE(offset >= 0 && offset <= total && elements * nq <= total - offset,
                 "P2 IB group exceeds table bounds");
    AFSI_REQUIRE(nx > 0 && ny > 0 && nz > 0, "invalid P2 MAC grid");
    return AFSI_OK;
}

extern "C" int32_t afsi_b200_p2_spread(const void* value, int64_t nodes, const int64_t* cells, int64_t elements,
                                       const void* N, int64_t nq, const void* W, const int64_t* base,
                                       const void* phi, int64_t total, int64_t offset, void* u0, void* u1, void* u2,
                                       int64_t nx, int64_t ny, int64_t nz, double volume, int32_t* status,
                                       int32_t dtype, afsi_stream_t stream) {
    int32_t rc = p2_check(elements, nq, total, offset, nx, ny, nz);
    if (rc) return rc;
    AFSI_REQUIRE(isfinite(volume) && volume > 0, "invalid P2 MAC grid");
    if (elements == 0) return AFSI_OK;
    AFSI_REQUIRE(value && cells && N && W && base && phi && u0 && u1 && u2, "null device pointer");
    P2Dims g{nx, ny, nz, total, offset, nq, nodes, elements};
    AFSI_DISPATCH(dtype, {
        return launch_spread_staged<T>(static_cast<const T*>(value), cells, static_cast<const T*>(N),
                                       static_cast<const T*>(W), base, static_cast<const T*>(phi),
                                       static_cast<T*>(u0), static_cast<T*>(u1), static_cast<T*>(u2), g, T(volume),
                                       status, staged_blocks(elements), stream);
    });
    return AFSI_OK;
}

template <bool Local>
static int32_t p2_gather(const void* u0, const void* u1, const void* u2, const int64_t* cells, int64_t elements,
                         const void* N, int64_t nq, const void* W, const int64_t* base, const void* phi,
                         int64_t total, int64_t offset, void* out, int64_t nodes, int64_t nx, int64_t ny,
                         int64_t nz, int32_t* status, int32_t dtype, afsi_stream_t stream) {
    int32_t rc = p2_check(elements, nq, total, offset, nx, ny, nz);
    if (rc) return rc;
    if (elements == 0) return AFSI_OK;
    AFSI_REQUIRE(u0 && u1 && u2 && cells && N && W && base && phi && out, "null device pointer");
    P2Dims g{nx, ny, nz, total, offset, nq, nodes, elements};
    AFSI_DISPATCH(dtype, {
        return launch_gather_staged<T, Local>(static_cast<const T*>(u0), static_cast<const T*>(u1),
                                              static_cast<const T*>(u2), cells, static_cast<const T*>(N),
                                              static_cast<const T*>(W), base, static_cast<const T*>(phi),
                                              static_cast<T*>(out), g, status, staged_blocks(elements), stream);
    });
    return AFSI_OK;
}

extern "C" int32_t afsi_b200_p2_gather_assemble(const void* u0, const void* u1, const void* u2,
                                                const int64_t* cells, int64_t elements, const void* N, int64_t nq,
                                                const void* W, const int64_t* base, const void* phi, int64_t total,
                                                int64_t offset, void* rhs, int64_t nodes, int64_t nx, int64_t ny,
                                                int64_t nz, int32_t* status, int32_t dtype, afsi_stream_t stream) {
    return p2_gather<false>(u0, u1, u2, cells, elements, N, nq, W, base, phi, total, offset, rhs, nodes, nx, ny, nz,
                            status, dtype, stream);
}

extern "C" int32_t afsi_b200_p2_gather_local(const void* u0, const void* u1, const void* u2, const int64_t* cells,
                                             int64_t elements, const void* N, int64_t nq, const void* W,
                                             const int64_t* base, const void* phi, int64_t total, int64_t offset,
                                             void* local, int64_t nx, int64_t ny, int64_t nz, int32_t* status,
                                             int32_t dtype, afsi_stream_t stream) {
    return p2_gather<true>(u0, u1, u2, cells, elements, N, nq, W, base, phi, total, offset, local, INT64_MAX, nx,
                           ny, nz, status, dtype, stream);
}

extern "C" int32_t afsi_b200_node_reduce(const void* local, int64_t slots, const int64_t* crow, const int64_t* slot,
                                         int64_t nodes, void* rhs, int32_t accumulate, int32_t* status,
                                         int32_t dtype, afsi_stream_t stream) {
    AFSI_REQUIRE(nodes >= 0 && slots >= 0, "invalid node reduction sizes");
    if (nodes == 0) return AFSI_OK;
    AFSI_REQUIRE(local && crow && slot && rhs, "null device pointer");
    AFSI_DISPATCH(dtype, {
        node_reduce_kernel<T><<<blocks_for(nodes, 256), 256, 0, stream>>>(
            static_cast<const T*>(local), slots, crow, slot, nodes, static_cast<T*>(rhs), accumulate, status);
    });
    return launched("node_reduce");
}
