// Consistent-mass Jacobi-PCG for the IB transfers on the B200.
//
// Solves M x = rhs for the (rows, cols) nodal block with the recurrence of
// mac/mass_solver.py:12-103 (and its graph form mac/mass_graph.py:118-225):
// one CG recurrence for all columns (every inner product over the whole
// block), z = r/diag, the breakdown guard on the curvature and rz, restart
// every recompute_every iterations, checks every check_every iterations (and
// at max_iterations), acceptance only on the true residual ||rhs - M x||.
//
// The reference reads device scalars on the host at every check; here the
// check itself runs on the device, so a whole solve is
//   begin   x = initial, ||rhs||, finiteness of rhs/initial, tol;
//   check   (iteration 0) r = rhs - M x, true norm, restart d = r/diag;
//   loop    spmv   Ad = M d, curvature d·Ad;
//           update alpha (the guard of _advance), x += alpha d, r -= alpha Ad,
//                  ||r||, r·(r/diag);
//           check  the rest of _advance and the reference's decision for this
//                  iteration: direction d = active ? r/diag + beta d : 0, or
//                  the true residual with its restart, or a stop (breakdown,
//                  converged, nonfinite true residual, out of iterations);
// with the loop a WHILE node of a CUDA graph whose body holds several iterations
// (loop_unroll) and whose last check ends it.  The caller reads the state once,
// at the end.  Every kernel is a no-op once the status leaves RUNNING, so a body
// or the stepped (graph-free) form may overrun.
//
// An iteration is a chain of three short kernels, bound by latency: the launch
// hand-over, the dependent loads and the reductions.  Therefore
//  * the inner products of spmv and update are left as one partial per block
//    and summed by every block of the kernel that needs them, in the same fixed
//    order (deterministic), instead of by the last block to arrive after a
//    fence and a counter; only begin and the true residual (once in tens of
//    iterations) still use the last block;
//  * a kernel writes no state word that its own blocks read (kBrokenNext and
//    kIterNext hand the values of update on to check);
//  * what does not depend on the iteration (the matrix's indices and values,
//    the diagonal) is loaded before the wait for the preceding kernel
//    (programmatic dependent launch);
//  * a turn of the WHILE node costs as much as two kernels, so one body runs
//    several iterations.
// P2 shell of 64,896 nodes and 1.61 M entries, three FP64 columns, 60
// iterations, one B200: 34.8 us per iteration before, 26.8 with these and 26.1
// with a row of d read by two loads.
//
// Element arithmetic is the reference's, operation for operation (the
// library is built with --fmad=false): z = r/diag, z + beta*d, x + alpha*d,
// r - alpha*Ad, products rounded in the element type before they are summed
// (in double).  Only the summation order of the inner products and of each
// CSR row differs from torch's.
#include "common.cuh"

namespace afsi {

enum PcgSlot : int {
    kRz = 0,         // rz of the current direction d
    kRzPending = 1,  // r·(r/diag) of the latest residual (kRz from the next spmv on)
    kCurvature = 2,
    kAlpha = 3,
    kRn = AFSI_PCG_RESIDUAL,  // ||r|| after the latest update
    kTol = AFSI_PCG_TOLERANCE,
    kActive = 6,
    kBroken = AFSI_PCG_BROKEN,
    kWorking = 8,
    kTrue = AFSI_PCG_TRUE_NORM,
    kIter = AFSI_PCG_ITERATIONS,
    kStatus = AFSI_PCG_STATUS,
    kRhsNorm = AFSI_PCG_RHS_NORM,
    kBrokenNext = 13,  // update -> check
    kIterNext = 14,    // update -> check
};

constexpr int kPcgThreads = 256;
constexpr int kPcgBlocks = 2048;  // grid cap; the partials hold 2 doubles per block
constexpr int kSpmvBlocks = 148 * 4;   // spmv: one wave (64 registers a thread)
constexpr int kUpdateBlocks = 148 * 4; // update, check: partials that a block sums in three loads per thread
constexpr int kRowLanes = 8;      // lanes per CSR row in the SpMV kernels
constexpr int kRowUnroll = 4;     // entries per lane whose loads are issued together

template <class T, class I>
struct Pcg {
    const int64_t* crow;
    const I* col;
    const T* val;
    const T* diag;
    const T* rhs;
    const T* init;
    T* x;
    T* r;
    T* d;
    T* Ad;
    double* state;
    double* partial;       // begin, true residual: two doubles per block
    double* curvature;     // spmv: one double per block
    double* norms;         // update: two doubles per block
    unsigned int* counter;
    int32_t spmv_blocks, update_blocks;
    int64_t rows;
    int32_t max_iterations, check_every, recompute_every, diag_per_row;
    double rtol, atol;
};

__device__ __forceinline__ bool running(const double* state) { return state[kStatus] == AFSI_PCG_RUNNING; }

// Diagonal entry of element i (row i / C).
template <int C, class T, class I>
__device__ __forceinline__ T diag_of(const Pcg<T, I>& p, int64_t i) {
    return p.diag[p.diag_per_row ? i / C : i];
}

// Adds this block's (a, b) to the partials; true in the one block that
// finishes last, whose thread 0 then holds the totals.
__device__ bool pcg_reduce(double a, double b, double* partial, unsigned int* counter, double* tot) {
    __shared__ double sh[2][kPcgThreads / 32];
    __shared__ bool last;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    a = warp_sum(a);
    b = warp_sum(b);
    if (lane == 0) {
        sh[0][warp] = a;
        sh[1][warp] = b;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double ta = 0.0, tb = 0.0;
        for (int w = 0; w < kPcgThreads / 32; ++w) {
            ta += sh[0][w];
            tb += sh[1][w];
        }
        partial[2 * blockIdx.x] = ta;
        partial[2 * blockIdx.x + 1] = tb;
        __threadfence();
        last = atomicAdd(counter, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return false;
    __threadfence();
    // thread t sums partials t, t + 256, ... ; then the same fixed tree as above
    double ta = 0.0, tb = 0.0;
    for (unsigned k = threadIdx.x; k < gridDim.x; k += kPcgThreads) {
        ta += __ldcg(partial + 2 * k);
        tb += __ldcg(partial + 2 * k + 1);
    }
    ta = warp_sum(ta);
    tb = warp_sum(tb);
    __syncthreads();
    if (lane == 0) {
        sh[0][warp] = ta;
        sh[1][warp] = tb;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        ta = 0.0;
        tb = 0.0;
        for (int w = 0; w < kPcgThreads / 32; ++w) {
            ta += sh[0][w];
            tb += sh[1][w];
        }
        tot[0] = ta;
        tot[1] = tb;
        *counter = 0u;
    }
    return true;
}

// Sums of `width` (1 or 2) doubles per block over `blocks` partials, in every
// thread of the calling block: thread t adds partials t, t + 256, ..., then a
// fixed tree.  The same order, and the same bits, in every block.
__device__ __forceinline__ void sum_blocks(const double* partial, int blocks, int width, double* tot) {
    __shared__ double sh[2][kPcgThreads / 32];
    double a = 0.0, b = 0.0;
    for (int k = threadIdx.x; k < blocks; k += kPcgThreads) {
        a += __ldcg(partial + width * k);
        if (width == 2) b += __ldcg(partial + 2 * k + 1);
    }
#pragma unroll
    for (int d = 16; d; d >>= 1) {
        a += __shfl_xor_sync(0xffffffffu, a, d);
        if (width == 2) b += __shfl_xor_sync(0xffffffffu, b, d);
    }
    if ((threadIdx.x & 31) == 0) {
        sh[0][threadIdx.x >> 5] = a;
        sh[1][threadIdx.x >> 5] = b;
    }
    __syncthreads();
    a = b = 0.0;
#pragma unroll
    for (int w = 0; w < kPcgThreads / 32; ++w) {
        a += sh[0][w];
        b += sh[1][w];
    }
    tot[0] = a;
    tot[1] = b;
}

// This block's (a, b) to its slot of the partials.
__device__ __forceinline__ void put_partial(double a, double b, double* partial, int width) {
    __shared__ double sh[2][kPcgThreads / 32];
    a = warp_sum(a);
    if (width == 2) b = warp_sum(b);
    if ((threadIdx.x & 31) == 0) {
        sh[0][threadIdx.x >> 5] = a;
        sh[1][threadIdx.x >> 5] = b;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        a = b = 0.0;
        for (int w = 0; w < kPcgThreads / 32; ++w) {
            a += sh[0][w];
            b += sh[1][w];
        }
        partial[width * blockIdx.x] = a;
        if (width == 2) partial[2 * blockIdx.x + 1] = b;
    }
}

// A lane's share of a CSR row: entries j, j + 8, ... < end, the first
// kRowUnroll of them loaded.
template <class T, class I>
struct RowHead {
    int64_t j, end;
    I c[kRowUnroll];
    T m[kRowUnroll];
};

template <class T, class I>
__device__ __forceinline__ void load_entries(const Pcg<T, I>& p, RowHead<T, I>& h) {
#pragma unroll
    for (int u = 0; u < kRowUnroll; ++u) {
        const int64_t j = h.j + u * kRowLanes;
        h.c[u] = j < h.end ? p.col[j] : I(0);
        h.m[u] = j < h.end ? p.val[j] : T(0);
    }
}

template <class T, class I>
__device__ __forceinline__ RowHead<T, I> row_head(const Pcg<T, I>& p, int64_t row, int sub) {
    RowHead<T, I> h;
    h.j = h.end = 0;
    if (row < p.rows) {
        h.j = p.crow[row] + sub;
        h.end = p.crow[row + 1];
    }
    load_entries(p, h);
    return h;
}

// One row of a (rows, C) block.  Three doubles are 24 bytes on an 8- or a
// 16-byte boundary: a pair and a single, two loads instead of three.  The
// gathers bound the SpMV (a line per lane and load): 26.8 -> 26.1 us per iteration
// of the solve above.
template <class T, int C>
__device__ __forceinline__ void load_block_row(const T* __restrict__ src, T out[C]) {
    if constexpr (sizeof(T) == 8 && C == 3) {
        const bool odd = (reinterpret_cast<uintptr_t>(src) & 8) != 0;
        const double2 pair = *reinterpret_cast<const double2*>(src + (odd ? 1 : 0));
        const double one = src[odd ? 0 : 2];
        out[0] = odd ? one : pair.x;
        out[1] = odd ? pair.x : pair.y;
        out[2] = odd ? pair.y : one;
    } else {
#pragma unroll
        for (int c = 0; c < C; ++c) out[c] = src[c];
    }
}

// (M v)[row, :] for the calling 8-lane group (every lane ends with the sums).
// A lane takes the row's entries sub, sub + 8, ... in order, kRowUnroll at a
// time with their index and value loads issued before any gather.
template <class T, int C, class I>
__device__ __forceinline__ void row_product(const Pcg<T, I>& p, const T* __restrict__ v, RowHead<T, I>& h, T* y) {
#pragma unroll
    for (int c = 0; c < C; ++c) y[c] = T(0);
    while (h.j < h.end) {
#pragma unroll
        for (int u = 0; u < kRowUnroll; ++u) {
            if (h.j + u * kRowLanes < h.end) {
                T vj[C];
                load_block_row<T, C>(v + int64_t(h.c[u]) * C, vj);
#pragma unroll
                for (int c = 0; c < C; ++c) y[c] = fma(h.m[u], vj[c], y[c]);
            }
        }
        h.j += kRowUnroll * kRowLanes;
        if (h.j < h.end) load_entries(p, h);
    }
#pragma unroll
    for (int s = kRowLanes / 2; s; s >>= 1) {
#pragma unroll
        for (int c = 0; c < C; ++c) y[c] += __shfl_xor_sync(0xffffffffu, y[c], s);
    }
}

// Column `sub` of the row sums (lane `sub` of a group owns that column).
template <class T, int C>
__device__ __forceinline__ T column(const T* y, int sub) {
    T yc = y[0];
#pragma unroll
    for (int c = 1; c < C; ++c)
        if (sub == c) yc = y[c];
    return yc;
}

// x = initial; ||rhs||; finiteness of rhs and initial; tol = max(atol, rtol ||rhs||)
// (mac/mass_solver.py:57-71).
template <class T, int C, class I>
__global__ void __launch_bounds__(kPcgThreads) pcg_begin_kernel(Pcg<T, I> p) {
    pdl_enter();
    double rr = 0.0, bad = 0.0;
    const int64_t total = p.rows * C;
    for (int64_t i = int64_t(blockIdx.x) * kPcgThreads + threadIdx.x; i < total;
         i += int64_t(gridDim.x) * kPcgThreads) {
        const T b = p.rhs[i], x0 = p.init[i];
        p.x[i] = x0;
        rr += double(b) * double(b);
        if (!isfinite(b) || !isfinite(x0)) bad += 1.0;
    }
    double tot[2];
    if (!pcg_reduce(rr, bad, p.partial, p.counter, tot) || threadIdx.x != 0) return;
    const double norm = sqrt(tot[0]);
    const double scaled = p.rtol * norm;
    double* s = p.state;
    s[kRhsNorm] = norm;
    s[kTol] = scaled > p.atol ? scaled : p.atol;
    s[kIter] = 0.0;
    s[kRn] = 0.0;
    s[kTrue] = 0.0;
    s[kActive] = 0.0;
    s[kBroken] = 0.0;
    s[kWorking] = 0.0;
    s[kRz] = 1.0;
    s[kRzPending] = 0.0;
    s[kStatus] = tot[1] == 0.0 ? AFSI_PCG_RUNNING : AFSI_PCG_BAD_INPUT;
}

// Ad = M d and the block's share of the curvature d·Ad.
template <class T, int C, class I>
__global__ void __launch_bounds__(kPcgThreads, 4) pcg_spmv_kernel(Pcg<T, I> p) {
    const int sub = threadIdx.x % kRowLanes;
    const int64_t groups = int64_t(gridDim.x) * (kPcgThreads / kRowLanes);
    const int64_t first = (int64_t(blockIdx.x) * kPcgThreads + threadIdx.x) / kRowLanes;
    const int64_t rounds = (p.rows + groups - 1) / groups;
    pdl_launch();
    RowHead<T, I> head = row_head(p, first, sub);
    pdl_wait();
    if (!running(p.state)) return;
    double curv = 0.0;
    for (int64_t k = 0; k < rounds; ++k) {
        const int64_t row = first + k * groups;
        RowHead<T, I> next;
        if (k + 1 < rounds) next = row_head(p, row + groups, sub);
        T y[C];
        row_product<T, C, I>(p, p.d, head, y);
        if (row < p.rows && sub < C) {
            const T yc = column<T, C>(y, sub);
            const int64_t i = row * C + sub;
            p.Ad[i] = yc;
            curv += double(p.d[i] * yc);
        }
        head = next;
    }
    put_partial(curv, 0.0, p.curvature, 1);
}

// The guard of _advance (mac/mass_solver.py:12-17) and alpha from the
// curvature's partials, in every block; x += alpha d, r -= alpha Ad and the
// block's shares of ||r||^2 and r·(r/diag).
template <class T, int C, class I>
__global__ void __launch_bounds__(kPcgThreads) pcg_update_kernel(Pcg<T, I> p) {
    const int64_t total = p.rows * C, stride = int64_t(gridDim.x) * kPcgThreads;
    const int64_t first = int64_t(blockIdx.x) * kPcgThreads + threadIdx.x;
    pdl_launch();
    T diag = first < total ? diag_of<C>(p, first) : T(1);
    pdl_wait();
    double* s = p.state;
    if (!running(s)) return;
    T x0 = T(0), d0 = T(0), r0 = T(0), a0 = T(0);
    if (first < total) {  // in flight during the sum
        x0 = p.x[first];
        d0 = p.d[first];
        r0 = p.r[first];
        a0 = p.Ad[first];
    }
    double curvature[2];
    sum_blocks(p.curvature, p.spmv_blocks, 1, curvature);
    const double pending = s[kRzPending];
    const bool active = s[kActive] != 0.0;
    const bool valid = isfinite(curvature[0]) && curvature[0] > 0 && isfinite(pending) && pending > 0;
    const bool broken = s[kBroken] != 0.0 || (active && !valid);
    const bool working = active && valid && !broken;
    const double step = working ? pending / curvature[0] : 0.0;
    const T alpha = T(step);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        s[kRz] = pending;
        s[kCurvature] = curvature[0];
        s[kBrokenNext] = broken ? 1.0 : 0.0;
        s[kWorking] = working ? 1.0 : 0.0;
        s[kAlpha] = step;
        s[kIterNext] = s[kIter] + 1.0;
    }
    double rr = 0.0, rz = 0.0;
    for (int64_t i = first; i < total; i += stride) {
        p.x[i] = x0 + alpha * d0;
        const T ri = r0 - alpha * a0;
        p.r[i] = ri;
        rr += double(ri) * double(ri);
        rz += double(ri * (ri / diag));
        const int64_t n = i + stride;
        if (n < total) {
            diag = diag_of<C>(p, n);
            x0 = p.x[n];
            d0 = p.d[n];
            r0 = p.r[n];
            a0 = p.Ad[n];
        }
    }
    put_partial(rr, rz, p.norms, 2);
}

enum CheckMode : int { kIdle = 0, kDirection = 1, kTrueResidual = 2 };

// What the reference does after iteration `it` (mac/mass_solver.py:85-102):
// nothing more (stopped), the direction update, or the true residual with a
// restart.  Breakdown at a check stops the solve before the true residual.
template <class T, class I>
__device__ __forceinline__ int check_mode(const Pcg<T, I>& p, int64_t it, bool broken, double rn, bool* breakdown) {
    *breakdown = false;
    if (it == 0) return kTrueResidual;
    const bool restart = it % p.recompute_every == 0;
    const bool last = it == p.max_iterations;
    if (!(restart || it % p.check_every == 0 || last)) return kDirection;
    if (broken) {
        *breakdown = true;
        return kIdle;
    }
    return (restart || rn <= p.state[kTol] || last) ? kTrueResidual : kDirection;
}

// The rest of _advance (mac/mass_solver.py:18-23) from the update's partials,
// in every block, and the decision step.  initial: the residual before the
// first iteration.  With `loop` set it also ends or continues the WHILE node of
// the solve graph.
template <class T, int C, class I>
__global__ void __launch_bounds__(kPcgThreads) pcg_check_kernel(Pcg<T, I> p, cudaGraphConditionalHandle handle,
                                                               int loop, int initial) {
    pdl_launch();
    const int64_t first_element = int64_t(blockIdx.x) * kPcgThreads + threadIdx.x;
    const T diag0 = first_element < p.rows * C ? diag_of<C>(p, first_element) : T(1);
    pdl_wait();
    double* s = p.state;
    const bool lead = blockIdx.x == 0 && threadIdx.x == 0;
    int mode = kIdle;
    bool breakdown = false, active = false;
    int64_t it = 0;
    double rz_next = 0.0;
    // one read per block: block 0 may write BREAKDOWN while other blocks start
    if (__syncthreads_or(threadIdx.x == 0 && running(s))) {
        double rn = 0.0;
        bool broken = false;
        if (!initial) {
            double tot[2];
            sum_blocks(p.norms, p.update_blocks, 2, tot);
            rn = sqrt(tot[0]);
            rz_next = tot[1];
            broken = s[kBrokenNext] != 0.0 || !isfinite(rn);
            active = s[kWorking] != 0.0 && rn > s[kTol];
            it = int64_t(s[kIterNext]);
            if (lead) {
                s[kRn] = rn;
                s[kBroken] = broken ? 1.0 : 0.0;
                s[kActive] = active ? 1.0 : 0.0;
                s[kRzPending] = rz_next;
                s[kIter] = double(it);
            }
        }
        mode = check_mode(p, it, broken, rn, &breakdown);
    }
    if (mode == kIdle) {
        // a block that reads BREAKDOWN already written by block 0 also lands here
        if (lead) {
            if (breakdown) s[kStatus] = AFSI_PCG_BREAKDOWN;
            if (loop) cudaGraphSetConditional(handle, 0u);
        }
        return;
    }
    const int64_t total = p.rows * C;
    if (mode == kDirection) {
        // _direction (mac/mass_solver.py:26-31)
        const T beta = T(rz_next / (active ? s[kRz] : 1.0));
        for (int64_t i = first_element; i < total; i += int64_t(gridDim.x) * kPcgThreads)
            p.d[i] = active ? p.r[i] / (i == first_element ? diag0 : diag_of<C>(p, i)) + beta * p.d[i] : T(0);
        if (lead && loop) cudaGraphSetConditional(handle, 1u);
        return;
    }
    // true residual r = rhs - M x and the restart d = r/diag
    // (mac/mass_solver.py:34-36,72-75,93-101)
    const int sub = threadIdx.x % kRowLanes;
    const int64_t groups = int64_t(gridDim.x) * (kPcgThreads / kRowLanes);
    const int64_t first = (int64_t(blockIdx.x) * kPcgThreads + threadIdx.x) / kRowLanes;
    const int64_t rounds = (p.rows + groups - 1) / groups;
    double rr = 0.0, rz = 0.0;
    for (int64_t k = 0; k < rounds; ++k) {
        const int64_t row = first + k * groups;
        T y[C];
        RowHead<T, I> head = row_head(p, row, sub);
        row_product<T, C, I>(p, p.x, head, y);
        if (row < p.rows && sub < C) {
            const int64_t i = row * C + sub;
            const T ri = p.rhs[i] - column<T, C>(y, sub);
            const T di = ri / diag_of<C>(p, i);
            p.r[i] = ri;
            p.d[i] = di;
            rr += double(ri) * double(ri);
            rz += double(ri * di);
        }
    }
    double tot[2];
    if (!pcg_reduce(rr, rz, p.partial, p.counter, tot) || threadIdx.x != 0) return;
    const double true_norm = sqrt(tot[0]);
    s[kTrue] = true_norm;
    int status = AFSI_PCG_RUNNING;
    if (it > 0 && !isfinite(true_norm))
        status = AFSI_PCG_NONFINITE;
    else if (true_norm <= s[kTol])
        status = AFSI_PCG_CONVERGED;
    else if (it >= p.max_iterations)
        status = AFSI_PCG_NOT_CONVERGED;
    s[kRzPending] = tot[1];
    s[kActive] = 1.0;
    s[kStatus] = status;
    if (loop) cudaGraphSetConditional(handle, status == AFSI_PCG_RUNNING ? 1u : 0u);
}

}  // namespace afsi

using namespace afsi;

namespace {

unsigned grid_for(int64_t threads) {
    const int64_t want = (threads + kPcgThreads - 1) / kPcgThreads;
    return unsigned(want < 1 ? 1 : (want < kPcgBlocks ? want : kPcgBlocks));
}

// One wave of blocks whose groups take the same number of rows, give or take one.
unsigned spmv_grid(int64_t rows) {
    constexpr int64_t per = kPcgThreads / kRowLanes;
    const int64_t rounds = (rows + kSpmvBlocks * per - 1) / (kSpmvBlocks * per);
    return unsigned((rows + rounds * per - 1) / (rounds * per));
}

unsigned update_grid(int64_t elements) {
    const int64_t rounds = (elements + int64_t(kUpdateBlocks) * kPcgThreads - 1) / (int64_t(kUpdateBlocks) * kPcgThreads);
    return unsigned((elements + rounds * kPcgThreads - 1) / (rounds * kPcgThreads));
}

// Iterations per turn of the WHILE node: a check interval (the solve stops at
// checks, so no iteration is wasted), within 2..8; 4 for other intervals, at
// most three no-op iterations at the end of a solve.
int loop_unroll(const afsi_pcg_plan& q) {
    const int u = q.check_every >= 2 && q.check_every <= 8 ? q.check_every : 4;
    return u < q.max_iterations ? u : q.max_iterations;
}

int32_t check_plan(const afsi_pcg_plan* plan) {
    AFSI_REQUIRE(plan, "null PCG plan");
    const afsi_pcg_plan& q = *plan;
    AFSI_REQUIRE(q.rows > 0 && q.cols >= 1 && q.cols <= 3, "PCG plan needs rows > 0 and 1 to 3 columns");
    AFSI_REQUIRE((q.col != nullptr) != (q.col32 != nullptr), "PCG plan needs exactly one of col and col32");
    AFSI_REQUIRE(q.crow && q.val && q.diagonal && q.rhs && q.initial && q.x && q.r && q.d && q.Ad && q.state &&
                     q.scratch,
                 "null PCG plan buffer");
    AFSI_REQUIRE(q.max_iterations >= 1 && q.check_every >= 1 && q.recompute_every >= 1,
                 "PCG iteration counts must be positive");
    AFSI_REQUIRE(q.rows <= (q.col32 ? int64_t(INT32_MAX) : (int64_t(1) << 40)), "PCG rows out of range");
    AFSI_REQUIRE(q.diagonal_per_row == 0 || q.diagonal_per_row == 1, "diagonal_per_row must be 0 or 1");
    return AFSI_OK;
}

template <class T, class I>
Pcg<T, I> view(const afsi_pcg_plan& q, int kind) {
    Pcg<T, I> p;
    p.crow = q.crow;
    if constexpr (sizeof(I) == 4)
        p.col = q.col32;
    else
        p.col = q.col;
    p.val = static_cast<const T*>(q.val);
    p.diag = static_cast<const T*>(q.diagonal);
    p.rhs = static_cast<const T*>(q.rhs);
    p.init = static_cast<const T*>(q.initial);
    p.x = static_cast<T*>(q.x);
    p.r = static_cast<T*>(q.r);
    p.d = static_cast<T*>(q.d);
    p.Ad = static_cast<T*>(q.Ad);
    p.state = q.state;
    p.partial = static_cast<double*>(q.scratch);
    p.counter = reinterpret_cast<unsigned int*>(static_cast<unsigned char*>(q.scratch) + kPcgBlocks * 16) + kind;
    p.curvature = p.partial + kPcgBlocks * 2 + 8;
    p.norms = p.curvature + kPcgBlocks;
    p.spmv_blocks = int32_t(spmv_grid(q.rows));
    p.update_blocks = int32_t(update_grid(q.rows * q.cols));
    p.rows = q.rows;
    p.max_iterations = q.max_iterations;
    p.check_every = q.check_every;
    p.recompute_every = q.recompute_every;
    p.diag_per_row = q.diagonal_per_row;
    p.rtol = q.rtol;
    p.atol = q.atol;
    return p;
}

enum Kind : int { kBegin = 0, kSpmv = 1, kUpdate = 2, kCheck = 3 };

template <class T, int C, class I>
int32_t begin(const afsi_pcg_plan& q, cudaStream_t stream) {
    int32_t rc = launch_pdl("pcg begin", pcg_begin_kernel<T, C, I>, dim3(grid_for(q.rows * C)), dim3(kPcgThreads),
                            0, stream, view<T, I>(q, kBegin));
    if (rc) return rc;
    return launch_pdl("pcg initial residual", pcg_check_kernel<T, C, I>, dim3(grid_for(q.rows * kRowLanes)),
                      dim3(kPcgThreads), 0, stream, view<T, I>(q, kCheck), cudaGraphConditionalHandle(0), 0, 1);
}

template <class T, int C, class I>
int32_t iteration(const afsi_pcg_plan& q, cudaStream_t stream, cudaGraphConditionalHandle handle, int loop) {
    int32_t rc = launch_pdl("pcg spmv", pcg_spmv_kernel<T, C, I>, dim3(spmv_grid(q.rows)), dim3(kPcgThreads), 0, stream,
                            view<T, I>(q, kSpmv));
    if (rc) return rc;
    rc = launch_pdl("pcg update", pcg_update_kernel<T, C, I>, dim3(update_grid(q.rows * C)), dim3(kPcgThreads), 0,
                    stream, view<T, I>(q, kUpdate));
    if (rc) return rc;
    return launch_pdl("pcg check", pcg_check_kernel<T, C, I>, dim3(update_grid(q.rows * C)), dim3(kPcgThreads), 0,
                      stream, view<T, I>(q, kCheck), handle, loop, 0);
}

// Returns EXPR evaluated with T, C and I bound to the plan's element type,
// column count and column-index type.
#define PCG_ONE(q, TT, CC, EXPR)                                     \
    if ((q).col32) {                                                 \
        using T = TT;                                                \
        constexpr int C = CC;                                        \
        using I = int32_t;                                           \
        return EXPR;                                                 \
    } else {                                                         \
        using T = TT;                                                \
        constexpr int C = CC;                                        \
        using I = int64_t;                                           \
        return EXPR;                                                 \
    }
#define PCG_DISPATCH(q, EXPR)                                                                 \
    switch ((q).dtype * 4 + (q).cols) {                                                       \
    case AFSI_F32 * 4 + 1: { PCG_ONE(q, float, 1, EXPR) }                                     \
    case AFSI_F32 * 4 + 2: { PCG_ONE(q, float, 2, EXPR) }                                     \
    case AFSI_F32 * 4 + 3: { PCG_ONE(q, float, 3, EXPR) }                                     \
    case AFSI_F64 * 4 + 1: { PCG_ONE(q, double, 1, EXPR) }                                    \
    case AFSI_F64 * 4 + 2: { PCG_ONE(q, double, 2, EXPR) }                                    \
    case AFSI_F64 * 4 + 3: { PCG_ONE(q, double, 3, EXPR) }                                    \
    default: return fail(AFSI_ERR_ARG, "unsupported PCG dtype code %d", int((q).dtype));      \
    }

struct PcgGraph {
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    cudaStream_t capture = nullptr;
};

void release(PcgGraph* g) {
    if (!g) return;
    if (g->exec) cudaGraphExecDestroy(g->exec);
    if (g->graph) cudaGraphDestroy(g->graph);
    if (g->capture) cudaStreamDestroy(g->capture);
    delete g;
}

}  // namespace

extern "C" int64_t afsi_b200_pcg_scratch_bytes(void) { return int64_t(kPcgBlocks) * 40 + 64; }

extern "C" int32_t afsi_b200_pcg_begin(const afsi_pcg_plan* plan, afsi_stream_t stream) {
    int32_t rc = check_plan(plan);
    if (rc) return rc;
    PCG_DISPATCH(*plan, (begin<T, C, I>(*plan, stream)));
}

extern "C" int32_t afsi_b200_pcg_iterations(const afsi_pcg_plan* plan, int32_t count, afsi_stream_t stream) {
    int32_t rc = check_plan(plan);
    if (rc) return rc;
    AFSI_REQUIRE(count >= 1, "PCG step count must be positive");
    auto one = [&]() -> int32_t {
        PCG_DISPATCH(*plan, (iteration<T, C, I>(*plan, stream, cudaGraphConditionalHandle(0), 0)));
    };
    for (int32_t k = 0; k < count && !rc; ++k) rc = one();
    return rc;
}

extern "C" int32_t afsi_b200_pcg_graph_create(const afsi_pcg_plan* plan, void** graph_out) {
    int32_t rc = check_plan(plan);
    if (rc) return rc;
    AFSI_REQUIRE(graph_out, "null PCG graph argument");
    *graph_out = nullptr;
    PcgGraph* g = new PcgGraph;
    cudaGraphConditionalHandle handle;
    cudaGraphNodeParams np = {};
    cudaGraphNode_t node;
    // the loop is entered once per launch; a solve that already stopped in
    // afsi_b200_pcg_begin passes through the body as no-ops
    if (cudaStreamCreateWithFlags(&g->capture, cudaStreamNonBlocking) != cudaSuccess ||
        cudaGraphCreate(&g->graph, 0) != cudaSuccess ||
        cudaGraphConditionalHandleCreate(&handle, g->graph, 1, cudaGraphCondAssignDefault) != cudaSuccess) {
        release(g);
        return fail(AFSI_ERR_CUDA, "PCG graph setup failed: %s", cudaGetErrorString(cudaGetLastError()));
    }
    np.type = cudaGraphNodeTypeConditional;
    np.conditional.handle = handle;
    np.conditional.type = cudaGraphCondTypeWhile;
    np.conditional.size = 1;
    if (cudaGraphAddNode(&node, g->graph, nullptr, 0, &np) != cudaSuccess) {
        release(g);
        return fail(AFSI_ERR_CUDA, "PCG conditional node failed: %s", cudaGetErrorString(cudaGetLastError()));
    }
    cudaGraph_t body = np.conditional.phGraph_out[0];
    if (cudaStreamBeginCaptureToGraph(g->capture, body, nullptr, nullptr, 0, cudaStreamCaptureModeRelaxed) !=
        cudaSuccess) {
        release(g);
        return fail(AFSI_ERR_CUDA, "PCG graph capture failed: %s", cudaGetErrorString(cudaGetLastError()));
    }
    auto body_launches = [&]() -> int32_t {
        PCG_DISPATCH(*plan, (iteration<T, C, I>(*plan, g->capture, handle, 1)));
    };
    for (int u = loop_unroll(*plan); u > 0 && !rc; --u) rc = body_launches();
    cudaGraph_t captured = nullptr;
    const cudaError_t end = cudaStreamEndCapture(g->capture, &captured);
    if (rc) {
        release(g);
        return rc;
    }
    if (end != cudaSuccess || cudaGraphInstantiate(&g->exec, g->graph, 0) != cudaSuccess) {
        release(g);
        return fail(AFSI_ERR_CUDA, "PCG graph instantiation failed: %s", cudaGetErrorString(cudaGetLastError()));
    }
    *graph_out = g;
    return AFSI_OK;
}

extern "C" int32_t afsi_b200_pcg_graph_launch(void* graph, afsi_stream_t stream) {
    AFSI_REQUIRE(graph, "null PCG graph");
    if (cudaGraphLaunch(static_cast<PcgGraph*>(graph)->exec, stream) != cudaSuccess)
        return fail(AFSI_ERR_CUDA, "PCG graph launch failed: %s", cudaGetErrorString(cudaGetLastError()));
    return AFSI_OK;
}

extern "C" int32_t afsi_b200_pcg_graph_destroy(void* graph) {
    release(static_cast<PcgGraph*>(graph));
    return AFSI_OK;
}
