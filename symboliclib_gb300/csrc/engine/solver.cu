// Batched preconditioned Krylov solves on the device, for the step
// after assembly: solving A x = b with the cloth system matrix the engine
// evaluates (reference examples/BaraffWitkin/implementation/cloth.cpp:96-111
// assembles A = M - h (D + h K) and b; examples/BaraffWitkin/main.cpp:56 keeps
// its lower triangle, which is what the engine's cloth workload outputs).
// Conjugate gradient needs A positive definite; the cloth matrices of a
// stretched and compressed sheet are symmetric but indefinite (negative
// diagonal entries occur), for which BiCGSTAB is provided.  The default
// preconditioner scales by 1 / |A_ii| (equal to Jacobi for a positive definite
// A; with the signed diagonal of an indefinite A, BiCGSTAB breaks down);
// BiCGSTAB can instead use block Jacobi with the exact inverses of the b x b
// diagonal blocks of one node's unknowns (b = 3 for the cloth: a vertex's x, y
// and z rows, which the cloth matrix stores n apart).
//
// The pattern (lower-triangle or full CSC) is turned once into a full CSR
// that names, per entry, its value in the engine's result buffer (or, with
// few sets, the values are copied into CSR order).  Each solve turns the values
// of all S systems into [value][set] order and
// iterates on vectors laid out [row][set], so threads along the set index
// read contiguous memory.  Per-set scalars (step lengths, dot products) live on
// the device; the host looks at the residuals every kCheck iterations.
//
// An iteration is three kernels (CG) or five (BiCGSTAB): the fewest with a
// grid-wide dot product between any two; the preconditioner is applied where
// its operand is made and accumulators are cleared by kernels that do not use
// them, so nothing else is launched.  Figures (GB300, cloth pattern
// 100 x 100: 30 k rows, 1.14 M entries): BiCGSTAB with 3 x 3 blocks, 8 sets, 143
// us an iteration with nine launches, two cleared buffers and an atomic
// addition per row, 65 so; CG, 8 sets, 69 -> 34; CG, one set, 65 -> 17.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <limits>
#include <string>
#include <vector>

#include "symgb.h"
#include "unit.hpp"

namespace {

constexpr int kThreads = 256;
constexpr unsigned kVectorThreads = 1024;  // threads per SM of a vector update
constexpr int kCheck = 16;  // iterations between host convergence checks

// Every kernel of an iteration is launched with programmatic stream
// serialisation: it is scheduled while its predecessor drains and waits here
// for the predecessor's writes, so the gap between two kernels is not paid.
// All of them wait before touching memory, so their order is the stream's;
// what an earlier step wrote is read through plain pointers (a const
// __restrict__ load is free to move above the wait).  The next kernel is let in
// only when a block's rows are done: let in at the start, its waiting blocks
// take the free slots, the rest go wherever slots come free first, and the
// uneven spread over the SMs costs more than the gap (30 k rows x 8 sets: CG
// 49 us an iteration, 36 so).
__device__ __forceinline__ void stepBegin() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
}
__device__ __forceinline__ void stepEnd() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// A block's threads over [row][set] vectors: `rows` rows at a time, thread t
// on set t % S of row t / S; a thread keeps its set from pass to pass, so it
// sums its part of a dot product in a register.
struct Place {
    unsigned width, s, r, rows;
    __device__ explicit Place(unsigned S)
        : width(S), s(threadIdx.x % S), r(threadIdx.x / S), rows(blockDim.x / S) {}
    __device__ bool active() const { return r < rows; }
};

// dst[s] += the sum of v over the block's threads of set s, one atomic
// addition per block and set (red: blockDim.x doubles).  Pairwise in shared
// memory: one atomic per thread, as before, serialised the block on S words.
__device__ __forceinline__ void blockSum(const Place& at, unsigned S, double v, double* red, double* __restrict__ dst) {
    __syncthreads();
    red[threadIdx.x] = v;
    for (unsigned rows = at.rows; rows > 1;) {
        const unsigned half = (rows + 1) / 2;
        __syncthreads();
        if (at.r < rows - half) red[threadIdx.x] += red[threadIdx.x + half * at.width];
        rows = half;
    }
    if (threadIdx.x < S) atomicAdd(&dst[threadIdx.x], red[threadIdx.x]);
}

// scalar(s) of the thread's set, evaluated once per block and set: a double
// division is ten FP64 instructions, as much as a row's whole update.
template <class F>
__device__ __forceinline__ double perSet(unsigned S, double* red, F scalar) {
    if (threadIdx.x < S) red[threadIdx.x] = scalar(threadIdx.x);
    __syncthreads();
    const double v = red[threadIdx.x % S];
    __syncthreads();
    return v;
}

__device__ __forceinline__ void clearSets(double* __restrict__ a, unsigned count) {
    if (a && blockIdx.x == 0)
        for (unsigned q = threadIdx.x; q < count; q += blockDim.x) a[q] = 0.0;
}

// vals[e * S + s] = in[s * nIn + e], or with `dst` vals[d * S + s] for the one
// or two CSR positions d of input entry e (dst[2 e], dst[2 e + 1], -1: none).
// Tiles of 64 entries x 32 sets through shared memory: reads run along the
// entries of a set, writes along the sets of an entry.  (Gathering by CSR
// position read 8 bytes of every 32-byte sector.)
constexpr unsigned kEntryTile = 64, kSetTile = 32;
__global__ void __launch_bounds__(kThreads) placeValues(const double* __restrict__ in, std::uint64_t nIn,
                                                        const std::int64_t* __restrict__ dst, unsigned S,
                                                        double* __restrict__ vals) {
    __shared__ double tile[kEntryTile][kSetTile + 1];
    const std::uint64_t e0 = (std::uint64_t)blockIdx.x * kEntryTile;
    const unsigned s0 = blockIdx.y * kSetTile, sets = min(kSetTile, S - s0);
    const unsigned entries = (unsigned)min((std::uint64_t)kEntryTile, nIn - e0);
    for (unsigned q = threadIdx.x; q < kEntryTile * sets; q += kThreads) {
        const unsigned e = q % kEntryTile, s = q / kEntryTile;
        if (e < entries) tile[e][s] = in[(std::uint64_t)(s0 + s) * nIn + e0 + e];
    }
    __syncthreads();
    for (unsigned q = threadIdx.x; q < entries * sets; q += kThreads) {
        const unsigned e = q / sets, s = q - e * sets;
        const double v = tile[e][s];
        if (!dst) {
            vals[(e0 + e) * S + s0 + s] = v;
            continue;
        }
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const std::int64_t d = dst[2 * (e0 + e) + k];
            if (d >= 0) vals[(std::uint64_t)d * S + s0 + s] = v;
        }
    }
}

// y = A z, d1 += w.y and, with d2, d2 += y.y; clears `zero` and `zero2` (S values each).
// `lanes` threads share a row, thread t on set t % width (width >= S), lane
// (t / width) % lanes of row t / (width lanes); width x lanes divides 32 where
// lanes > 1.  `entry` gives a CSR entry's column and, SHARED, the index of its
// value: both entries of a symmetric pair read one value (30 k rows x 16 sets:
// 147 -> 75 MB, CG 92 -> 76 us an iteration).  Otherwise the values are in
// CSR order.
// Full rows of threads are bound by the FP64 pipe: 2 x nnz x S flops at 1.25
// TFLOP/s (14.6 us for 30 k rows, 1.14 M entries, 8 sets; the kernel takes
// 19.6).  With !WIDE all the chip's 2048 threads per SM are resident (32
// registers): at 40 the last 3 % of the blocks of that size formed a second
// wave, a third of the time.  WIDE is for systems that leave SMs idle, where a
// row's chain of loads is the time: more lanes, twice the loads in flight.
template <bool SHARED, bool WIDE>
__global__ void __launch_bounds__(kThreads, WIDE ? 4 : 2048 / kThreads)
    spmv(const std::int64_t* __restrict__ rowPtr, const uint2* __restrict__ entry, const double* __restrict__ vals,
         const double* z, std::uint64_t n, unsigned S, unsigned width, unsigned lanes, const double* w, double* y,
         double* d1, double* d2, double* zero, double* zero2) {
    extern __shared__ double red[];
    stepBegin();
    clearSets(zero, S);
    clearSets(zero2, S);
    const Place at(width);
    const unsigned l = at.r % lanes, r = at.r / lanes, rows = at.rows / lanes;
    double a = 0.0, c = 0.0;
    for (std::uint64_t base = (std::uint64_t)blockIdx.x * rows; base < n; base += (std::uint64_t)gridDim.x * rows) {
        const std::uint64_t i = base + r;
        const bool mine = r < rows && i < n && at.s < S;
        double acc = 0.0;
        if (mine) {
            const std::int64_t e0 = rowPtr[i] + l;
            const uint2* pe = entry + e0;
            const double* pv = SHARED ? vals + at.s : vals + (std::uint64_t)e0 * S + at.s;
            const double* zs = z + at.s;
#pragma unroll(WIDE ? 4 : 2)
            for (int left = (int)(rowPtr[i + 1] - e0); left > 0; left -= (int)lanes, pe += lanes) {
                const uint2 q = *pe;
                const double v = SHARED ? pv[(std::uint64_t)q.y * S] : *pv;
                acc = fma(v, zs[(std::uint64_t)q.x * S], acc);
                if (!SHARED) pv += (std::uint64_t)lanes * S;
            }
        }
        for (unsigned k = lanes / 2; k > 0; k >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, k * width);
        if (mine && l == 0) {
            y[i * S + at.s] = acc;
            a = fma(acc, w[i * S + at.s], a);
            if (d2) c = fma(acc, acc, c);
        }
    }
    stepEnd();
    blockSum(at, S, a, red, d1);
    if (d2) blockSum(at, S, c, red, d2);
}

// ---------------------------------------------------------------- conjugate gradient
// Scalars per set: rz (by iteration parity), pq, rr, bb.

// Start: x = 0, r = b, p = r / diag; rz = r.p, bb = b.b.
__global__ void __launch_bounds__(kThreads) cgStart(const double* __restrict__ b, const double* __restrict__ vals,
                                                    const std::int64_t* __restrict__ diagPos, std::uint64_t n,
                                                    unsigned S, double* __restrict__ x, double* __restrict__ r,
                                                    double* __restrict__ p, double* __restrict__ invDiag,
                                                    double* __restrict__ rz, double* __restrict__ bb) {
    extern __shared__ double red[];
    const Place at(S);
    double vrz = 0.0, vbb = 0.0;
    for (std::uint64_t i = (std::uint64_t)blockIdx.x * at.rows + at.r; at.active() && i < n;
         i += (std::uint64_t)gridDim.x * at.rows) {
        const std::uint64_t t = i * S + at.s;
        const double bi = b[(std::uint64_t)at.s * n + i];
        const double d = diagPos[i] >= 0 ? vals[(std::uint64_t)diagPos[i] * S + at.s] : 0.0;
        const double inv = d != 0.0 ? 1.0 / fabs(d) : 1.0;
        x[t] = 0.0;
        r[t] = bi;
        p[t] = bi * inv;
        invDiag[t] = inv;
        vrz = fma(bi * bi, inv, vrz);
        vbb = fma(bi, bi, vbb);
    }
    blockSum(at, S, vrz, red, rz);
    blockSum(at, S, vbb, red, bb);
}

// alpha = rz / pq; x += alpha p; r -= alpha q; rzNew += r.(r / diag); rr += r.r
__global__ void __launch_bounds__(kThreads) cgUpdate(const double* p, const double* q,
                                                     const double* invDiag, std::uint64_t n, unsigned S,
                                                     const double* rz, const double* pq,
                                                     double* x, double* r,
                                                     double* rzNew, double* rr) {
    extern __shared__ double red[];
    stepBegin();
    const Place at(S);
    const double alpha = perSet(S, red, [&](unsigned s) { return pq[s] != 0.0 ? rz[s] / pq[s] : 0.0; });
    double a = 0.0, c = 0.0;
    for (std::uint64_t i = (std::uint64_t)blockIdx.x * at.rows + at.r; at.active() && i < n;
         i += (std::uint64_t)gridDim.x * at.rows) {
        const std::uint64_t t = i * S + at.s;
        const double xi = fma(alpha, p[t], x[t]), ri = fma(-alpha, q[t], r[t]), di = invDiag[t];
        x[t] = xi;
        r[t] = ri;
        const double r2 = ri * ri;
        a = fma(r2, di, a);
        c += r2;
    }
    stepEnd();
    blockSum(at, S, a, red, rzNew);
    blockSum(at, S, c, red, rr);
}

// p = r / diag + beta p with beta = rzNew / rz; clears `zero` (S values)
__global__ void __launch_bounds__(kThreads) cgDirection(const double* r,
                                                        const double* invDiag, std::uint64_t n,
                                                        unsigned S, const double* rz,
                                                        const double* rzNew, double* p,
                                                        double* zero) {
    extern __shared__ double red[];
    stepBegin();
    clearSets(zero, S);
    const Place at(S);
    const double beta = perSet(S, red, [&](unsigned s) { return rz[s] != 0.0 ? rzNew[s] / rz[s] : 0.0; });
    for (std::uint64_t i = (std::uint64_t)blockIdx.x * at.rows + at.r; at.active() && i < n;
         i += (std::uint64_t)gridDim.x * at.rows) {
        const std::uint64_t t = i * S + at.s;
        p[t] = fma(beta, p[t], r[t] * invDiag[t]);
    }
    stepEnd();
}

// out[s * n + i] = x[i * S + s]
__global__ void transposeSets(const double* __restrict__ x, std::uint64_t n, unsigned S, double* __restrict__ out) {
    const std::uint64_t t = (std::uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n * S) return;
    const std::uint64_t s = t / n, i = t - s * n;
    out[t] = x[i * S + s];
}

// ---------------------------------------------------------------- BiCGSTAB
// Right-preconditioned BiCGSTAB (van der Vorst), the preconditioner a block
// diagonal of B x B inverses M^-1 (B = 1: 1 / |A_ii|).  Five kernels an
// iteration, one between any two dot products: direction, product, half
// step, product, finish.  Scalars per set: rho (two slots: current and, until
// the direction has read it, previous; then the next one's sum), rv, ts, tt,
// rr, bb, alpha, omega.

// x = 0, r = rhat = b, p = v = 0, invDiag = 1 / |A_ii|; rho = bb = b.b, previous rho = alpha = omega = 1
__global__ void __launch_bounds__(kThreads) bStart(const double* __restrict__ b, const double* __restrict__ vals,
                                                   const std::int64_t* __restrict__ diagPos, std::uint64_t n,
                                                   unsigned S, double* __restrict__ x, double* __restrict__ r,
                                                   double* __restrict__ rhat, double* __restrict__ p,
                                                   double* __restrict__ v, double* __restrict__ invDiag,
                                                   double* __restrict__ rho, double* __restrict__ rhoPrev,
                                                   double* __restrict__ alpha, double* __restrict__ omega,
                                                   double* __restrict__ bb) {
    extern __shared__ double red[];
    const Place at(S);
    if (blockIdx.x == 0 && threadIdx.x < S) rhoPrev[at.s] = alpha[at.s] = omega[at.s] = 1.0;
    double vbb = 0.0;
    for (std::uint64_t i = (std::uint64_t)blockIdx.x * at.rows + at.r; at.active() && i < n;
         i += (std::uint64_t)gridDim.x * at.rows) {
        const std::uint64_t t = i * S + at.s;
        const double bi = b[(std::uint64_t)at.s * n + i];
        const double d = diagPos[i] >= 0 ? vals[(std::uint64_t)diagPos[i] * S + at.s] : 0.0;
        x[t] = 0.0;
        r[t] = bi;
        rhat[t] = bi;
        p[t] = 0.0;
        v[t] = 0.0;
        invDiag[t] = d != 0.0 ? 1.0 / fabs(d) : 1.0;
        vbb = fma(bi, bi, vbb);
    }
    blockSum(at, S, vbb, red, rho);
    blockSum(at, S, vbb, red, bb);
}

// omega = ts / tt; x += alpha ph + omega sh; r = s - omega t; rhoNext += rhat.r; rr += r.r
__global__ void __launch_bounds__(kThreads) bFinishStep(
    const double* ph, const double* sh, const double* sv,
    const double* tv, const double* rhat, std::uint64_t n, unsigned S,
    const double* alpha, const double* ts, const double* tt,
    double* omega, double* x, double* r, double* rhoNext,
    double* rr) {
    extern __shared__ double red[];
    stepBegin();
    const Place at(S);
    const double om = perSet(S, red, [&](unsigned s) { return tt[s] != 0.0 ? ts[s] / tt[s] : 0.0; }), al = alpha[at.s];
    if (blockIdx.x == 0 && threadIdx.x < S) omega[at.s] = om;
    double a = 0.0, c = 0.0;
    for (std::uint64_t i = (std::uint64_t)blockIdx.x * at.rows + at.r; at.active() && i < n;
         i += (std::uint64_t)gridDim.x * at.rows) {
        const std::uint64_t t = i * S + at.s;
        const double xi = fma(om, sh[t], fma(al, ph[t], x[t])), ri = fma(-om, tv[t], sv[t]), hi = rhat[t];
        x[t] = xi;
        r[t] = ri;
        a = fma(hi, ri, a);
        c = fma(ri, ri, c);
    }
    stepEnd();
    blockSum(at, S, a, red, rhoNext);
    blockSum(at, S, c, red, rr);
}

// ---------------------------------------------------------------- block Jacobi
// Blocks of B unknowns: block j holds rows j * B + a (stride 1, unknowns of one
// node stored together) or j + a * stride (stride n / B, each coordinate's
// unknowns stored together, as the cloth matrix orders them).

__device__ __forceinline__ std::uint64_t blockRow(std::uint64_t j, int a, int B, std::uint64_t stride) {
    return stride == 1 ? j * (std::uint64_t)B + (std::uint64_t)a : j + (std::uint64_t)a * stride;
}

// inv[(j * B * B + a * B + c) * S + s] = (A_jj^-1)[a][c] of set s, by Gauss-Jordan
// elimination with partial pivoting; a block with a zero pivot takes the
// inverse of its absolute diagonal instead (the scaled-Jacobi fallback).
template <int B>
__global__ void blockInvert(const double* __restrict__ vals, const std::int64_t* __restrict__ pos, std::uint64_t nb,
                            unsigned S, double* __restrict__ inv) {
    const std::uint64_t t = (std::uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nb * S) return;
    const std::uint64_t j = t / S;
    const unsigned s = (unsigned)(t - j * S);
    double m[B][2 * B];
#pragma unroll
    for (int a = 0; a < B; ++a)
#pragma unroll
        for (int c = 0; c < B; ++c) {
            const std::int64_t e = pos[j * B * B + a * B + c];
            m[a][c] = e >= 0 ? vals[(std::uint64_t)e * S + s] : 0.0;
            m[a][B + c] = a == c ? 1.0 : 0.0;
        }
    bool singular = false;
#pragma unroll
    for (int c = 0; c < B; ++c) {
        int piv = c;
#pragma unroll
        for (int a = c + 1; a < B; ++a)
            if (fabs(m[a][c]) > fabs(m[piv][c])) piv = a;
        if (m[piv][c] == 0.0) {
            singular = true;
            break;
        }
#pragma unroll
        for (int q = 0; q < 2 * B; ++q) {
            const double tmp = m[c][q];
            m[c][q] = m[piv][q];
            m[piv][q] = tmp;
        }
        const double d = 1.0 / m[c][c];
#pragma unroll
        for (int q = 0; q < 2 * B; ++q) m[c][q] *= d;
#pragma unroll
        for (int a = 0; a < B; ++a)
            if (a != c) {
                const double f = m[a][c];
#pragma unroll
                for (int q = 0; q < 2 * B; ++q) m[a][q] = fma(-f, m[c][q], m[a][q]);
            }
    }
#pragma unroll
    for (int a = 0; a < B; ++a)
#pragma unroll
        for (int c = 0; c < B; ++c) {
            double v;
            if (!singular) {
                v = m[a][B + c];
            } else {
                const std::int64_t e = pos[j * B * B + a * B + a];
                const double d = e >= 0 ? vals[(std::uint64_t)e * S + s] : 0.0;
                v = a == c ? (d != 0.0 ? 1.0 / fabs(d) : 1.0) : 0.0;
            }
            inv[(j * B * B + a * B + c) * S + s] = v;
        }
}

// out rows of block j = M_j^-1 (in rows of block j)
template <int B>
__device__ __forceinline__ void applyBlock(const double* inv, std::uint64_t j, unsigned S, unsigned s,
                                           const double (&in)[B], double (&out)[B]) {
#pragma unroll
    for (int a = 0; a < B; ++a) {
        double acc = 0.0;
#pragma unroll
        for (int c = 0; c < B; ++c) acc = fma(inv[(j * B * B + a * B + c) * S + s], in[c], acc);
        out[a] = acc;
    }
}

// p = r + beta (p - omega v), beta = (rho / rhoPrev) (alpha / omega); ph =
// M^-1 p; clears rv, ts, tt, rr (`zero`, 4 S values).  One thread per block
// of B rows, so p never goes through memory before M^-1.
template <int B>
__global__ void __launch_bounds__(kThreads) bDirection(const double* r, const double* v,
                                                       const double* inv, std::uint64_t nb,
                                                       std::uint64_t stride, unsigned S,
                                                       const double* rho,
                                                       const double* rhoPrev,
                                                       const double* alpha,
                                                       const double* omega, double* p,
                                                       double* ph, double* zero) {
    extern __shared__ double red[];
    stepBegin();
    clearSets(zero, 4 * S);
    const Place at(S);
    const double om = omega[at.s];
    const double beta = perSet(S, red, [&](unsigned s) {
        const double den = rhoPrev[s] * omega[s];
        return den != 0.0 ? (rho[s] * alpha[s]) / den : 0.0;
    });
    for (std::uint64_t j = (std::uint64_t)blockIdx.x * at.rows + at.r; at.active() && j < nb;
         j += (std::uint64_t)gridDim.x * at.rows) {
        double pi[B], o[B];
#pragma unroll
        for (int a = 0; a < B; ++a) {
            const std::uint64_t t = blockRow(j, a, B, stride) * S + at.s;
            pi[a] = fma(beta, fma(-om, v[t], p[t]), r[t]);
        }
        applyBlock<B>(inv, j, S, at.s, pi, o);
#pragma unroll
        for (int a = 0; a < B; ++a) {
            const std::uint64_t t = blockRow(j, a, B, stride) * S + at.s;
            p[t] = pi[a];
            ph[t] = o[a];
        }
    }
    stepEnd();
}

// alpha = rho / rv; s = r - alpha v; sh = M^-1 s
template <int B>
__global__ void __launch_bounds__(kThreads) bHalf(const double* r, const double* v,
                                                  const double* inv, std::uint64_t nb,
                                                  std::uint64_t stride, unsigned S, const double* rho,
                                                  const double* rv, double* alpha,
                                                  double* sv, double* sh) {
    extern __shared__ double red[];
    stepBegin();
    const Place at(S);
    const double al = perSet(S, red, [&](unsigned s) { return rv[s] != 0.0 ? rho[s] / rv[s] : 0.0; });
    if (blockIdx.x == 0 && threadIdx.x < S) alpha[at.s] = al;
    for (std::uint64_t j = (std::uint64_t)blockIdx.x * at.rows + at.r; at.active() && j < nb;
         j += (std::uint64_t)gridDim.x * at.rows) {
        double si[B], o[B];
#pragma unroll
        for (int a = 0; a < B; ++a) {
            const std::uint64_t t = blockRow(j, a, B, stride) * S + at.s;
            si[a] = fma(-al, v[t], r[t]);
        }
        applyBlock<B>(inv, j, S, at.s, si, o);
#pragma unroll
        for (int a = 0; a < B; ++a) {
            const std::uint64_t t = blockRow(j, a, B, stride) * S + at.s;
            sv[t] = si[a];
            sh[t] = o[a];
        }
    }
    stepEnd();
}

unsigned blocksFor(std::uint64_t work) { return (unsigned)((work + kThreads - 1) / kThreads); }

void blockInvertLaunch(int B, const double* vals, const std::int64_t* pos, std::uint64_t nb, unsigned S, double* inv,
                       cudaStream_t st) {
    const unsigned g = blocksFor(nb * S);
    switch (B) {
        case 2: blockInvert<2><<<g, kThreads, 0, st>>>(vals, pos, nb, S, inv); break;
        case 3: blockInvert<3><<<g, kThreads, 0, st>>>(vals, pos, nb, S, inv); break;
        default: blockInvert<4><<<g, kThreads, 0, st>>>(vals, pos, nb, S, inv); break;
    }
}

// Launches an iteration's kernel with programmatic stream serialisation.
template <class... P, class... A>
void launchStep(void (*fn)(P...), unsigned grid, unsigned block, std::size_t smem, cudaStream_t st, A... args) {
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, fn, static_cast<P>(args)...);
}

}  // namespace

struct symgb_solver {
    std::uint64_t n = 0, nnzIn = 0, nnzFull = 0;
    unsigned S = 1;
    bool shared = false;  // both entries of a symmetric pair read one value (spmv)
    symgb::engine::DevBuf<std::int64_t> rowPtr, dst, diagPos;
    symgb::engine::DevBuf<uint2> entry;  // CSR: column, value index
    symgb::engine::DevBuf<double> vals, x, r, p, q, invDiag, scalars, rhat, v, ph, sv, sh, t;
    double* hostScalars = nullptr;  // pinned copy of rr and bb
    unsigned smCount = 1;
    unsigned threads = kThreads;  // per block: rows of S sets, as few idle threads as possible
    // Blocks of a launch over `rows` rows, `width` threads to a row's sets and
    // `lanes` sharing a row: as many passes as `perSm` threads per SM need,
    // the rows spread evenly.
    unsigned blocks(std::uint64_t rows, unsigned perSm, unsigned width, unsigned lanes) const {
        const std::uint64_t per = threads / width / lanes, tiles = (rows + per - 1) / per;
        const std::uint64_t most = (std::uint64_t)smCount * (perSm / threads), passes = (tiles + most - 1) / most;
        return (unsigned)((tiles + passes - 1) / passes);
    }
    // Vector updates: half the threads, so that the sums at a block's end and
    // the scalars at its start are paid for half as often.
    unsigned vectorBlocks(std::uint64_t rows) const { return blocks(rows, kVectorThreads, S, 1); }
    std::size_t sharedBytes() const { return threads * sizeof(double); }
    // Host copy of the full CSR (block positions) and the block preconditioner.
    std::vector<std::int64_t> rowPtrHost;
    std::vector<int> colHost;
    std::vector<unsigned> valueHost;  // value index per entry (shared values)
    int block = 1;                  // unknowns per block (1: scaled Jacobi)
    std::uint64_t blockStride = 1;  // 1: contiguous blocks; n / block: one unknown per coordinate group
    symgb::engine::DevBuf<std::int64_t> blockPos;
    symgb::engine::DevBuf<double> blockInv;
    ~symgb_solver() {
        if (hostScalars) cudaFreeHost(hostScalars);
    }
};

extern "C" {

int symgb_solver_create(int64_t n, const int64_t* col_ptr, const int32_t* row_idx, int lower_only, int num_sets,
                    symgb_solver_t* out) {
    using symgb::engine::setLastError;
    if (!out || !col_ptr || n < 1 || num_sets < 1 || num_sets > kThreads)
        return setLastError(SYMGB_ERR_ARGUMENT, "solver: bad argument (num_sets 1..256)");
    const std::uint64_t nnzIn = (std::uint64_t)col_ptr[n];
    if (nnzIn && !row_idx) return setLastError(SYMGB_ERR_ARGUMENT, "solver: null row indices");
    // Full CSR of the symmetric matrix, entry <-> input value.
    std::vector<std::vector<std::pair<int, std::int64_t>>> rows((std::size_t)n);
    std::vector<std::int64_t> diag((std::size_t)n, -1);
    for (std::int64_t j = 0; j < n; ++j) {
        if (col_ptr[j] > col_ptr[j + 1]) return setLastError(SYMGB_ERR_ARGUMENT, "solver: column pointers decrease");
        for (std::int64_t e = col_ptr[j]; e < col_ptr[j + 1]; ++e) {
            const int i = row_idx[e];
            if (i < 0 || i >= n) return setLastError(SYMGB_ERR_ARGUMENT, "solver: row index out of range");
            if (lower_only && i < j) return setLastError(SYMGB_ERR_ARGUMENT, "solver: entry above the diagonal");
            rows[(std::size_t)i].push_back({(int)j, e});
            if (i != j && lower_only) rows[(std::size_t)j].push_back({i, e});
        }
    }
    // Values are shared where a value's sets fill 32-byte sectors (4 sets up);
    // below, reading them in CSR order matters more than their number.
    const bool shared = num_sets >= 4 && nnzIn <= 0xffffffffull;
    // diag[i]: the value position of entry (i, i), -1 if the pattern has none
    std::vector<std::int64_t> rowPtr(1, 0), dst(2 * nnzIn, -1);
    std::vector<int> col;
    std::vector<uint2> entry;
    for (std::size_t i = 0; i < rows.size(); ++i) {
        auto& rw = rows[i];
        std::sort(rw.begin(), rw.end());
        diag[i] = -1;
        for (auto& c : rw) {
            if (c.first == (int)i) diag[i] = shared ? c.second : (std::int64_t)col.size();
            std::int64_t* d = &dst[2 * (std::size_t)c.second];
            d[d[0] < 0 ? 0 : 1] = (std::int64_t)col.size();
            col.push_back(c.first);
            entry.push_back(make_uint2((unsigned)c.first, (unsigned)c.second));
        }
        rowPtr.push_back((std::int64_t)col.size());
    }
    auto* s = new symgb_solver();
    s->n = (std::uint64_t)n;
    s->nnzIn = nnzIn;
    s->nnzFull = col.size();
    s->S = (unsigned)num_sets;
    s->shared = shared;
    // Block size: the multiple of 32 whose rows of S sets leave the smallest
    // share of its threads idle; 128 (8 blocks to each wave's uneven end
    // instead of 16) where several do.
    double best = 0.0;
    for (unsigned t = 128; t <= (unsigned)kThreads; t += 32) {
        const double used = (double)(t / s->S * s->S) / t;
        if (used > best) best = used, s->threads = t;
    }
    int device = 0, sms = 1;
    cudaGetDevice(&device);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    s->smCount = (unsigned)std::max(1, sms);
    const std::uint64_t work = s->n * s->S;
    auto fail = [&](const char* what) {
        delete s;
        return setLastError(SYMGB_ERR_NOMEM, std::string("solver: ") + what);
    };
    if (s->rowPtr.alloc(rowPtr.size()) || (!shared && s->dst.alloc(dst.size())) || s->entry.alloc(entry.size()) ||
        s->diagPos.alloc(diag.size()) || s->vals.alloc((shared ? nnzIn : s->nnzFull) * s->S) || s->x.alloc(work) || s->r.alloc(work) ||
        s->p.alloc(work) || s->q.alloc(work) || s->invDiag.alloc(work) || s->scalars.alloc(16 * (std::size_t)s->S))
        return fail("device allocation failed");
    if (cudaMallocHost(&s->hostScalars, 2 * s->S * sizeof(double)) != cudaSuccess) return fail("pinned allocation failed");
    cudaMemcpy(s->rowPtr.ptr, rowPtr.data(), rowPtr.size() * 8, cudaMemcpyHostToDevice);
    if (!shared && !dst.empty()) cudaMemcpy(s->dst.ptr, dst.data(), dst.size() * 8, cudaMemcpyHostToDevice);
    if (!entry.empty()) cudaMemcpy(s->entry.ptr, entry.data(), entry.size() * sizeof(uint2), cudaMemcpyHostToDevice);
    cudaMemcpy(s->diagPos.ptr, diag.data(), diag.size() * 8, cudaMemcpyHostToDevice);
    if (cudaGetLastError() != cudaSuccess) return fail("upload failed");
    s->rowPtrHost = std::move(rowPtr);
    s->colHost = std::move(col);
    if (shared) {
        s->valueHost.reserve(entry.size());
        for (const uint2& q : entry) s->valueHost.push_back(q.y);
    }
    *out = s;
    return SYMGB_OK;
}

int symgb_solver_set_block_preconditioner(symgb_solver_t s, int block_size, int64_t stride) {
    using symgb::engine::setLastError;
    if (!s || block_size < 1 || block_size > 4) return setLastError(SYMGB_ERR_ARGUMENT, "solver: block size 1..4");
    if (block_size == 1) {
        s->block = 1;
        return SYMGB_OK;
    }
    const std::uint64_t n = s->n, B = (std::uint64_t)block_size;
    if (n % B) return setLastError(SYMGB_ERR_ARGUMENT, "solver: unknowns not a multiple of the block size");
    if (stride != 1 && (std::uint64_t)stride * B != n)
        return setLastError(SYMGB_ERR_ARGUMENT, "solver: stride must be 1 or n / block_size");
    const std::uint64_t nb = n / B;
    auto row = [&](std::uint64_t j, std::uint64_t a) { return stride == 1 ? j * B + a : j + a * (std::uint64_t)stride; };
    std::vector<std::int64_t> pos(nb * B * B, -1);
    for (std::uint64_t j = 0; j < nb; ++j)
        for (std::uint64_t a = 0; a < B; ++a) {
            const std::uint64_t r = row(j, a);
            const int* b = s->colHost.data() + s->rowPtrHost[r];
            const int* e = s->colHost.data() + s->rowPtrHost[r + 1];
            for (std::uint64_t c = 0; c < B; ++c) {
                const int* f = std::lower_bound(b, e, (int)row(j, c));
                if (f != e && *f == (int)row(j, c)) {
                    const std::size_t at = (std::size_t)(f - s->colHost.data());
                    pos[(j * B + a) * B + c] = s->shared ? (std::int64_t)s->valueHost[at] : (std::int64_t)at;
                }
            }
        }
    if (s->blockPos.alloc(pos.size()) || s->blockInv.alloc(pos.size() * s->S))
        return setLastError(SYMGB_ERR_NOMEM, "solver: device allocation failed");
    if (cudaMemcpy(s->blockPos.ptr, pos.data(), pos.size() * 8, cudaMemcpyHostToDevice) != cudaSuccess)
        return setLastError(SYMGB_ERR_CUDA, "solver: upload failed");
    s->block = block_size;
    s->blockStride = (std::uint64_t)stride;
    return SYMGB_OK;
}

// Values of every system, sets innermost; a matrix without entries is refused.
static int place(symgb_solver_t s, const double* values, cudaStream_t st) {
    if (!s->nnzIn) return symgb::engine::setLastError(SYMGB_ERR_CUDA, "solver: the matrix has no entries");
    const dim3 grid((unsigned)((s->nnzIn + kEntryTile - 1) / kEntryTile), (s->S + kSetTile - 1) / kSetTile);
    placeValues<<<grid, kThreads, 0, st>>>(values, s->nnzIn, s->shared ? nullptr : s->dst.ptr, s->S, s->vals.ptr);
    return SYMGB_OK;
}

// y = A z with its dot products (spmv).  Threads to a row: 8 / S while the
// sets alone would leave a warp's reads scattered over its 32 rows; more, up
// to a warp, while the threads fill less than half the chip (rows of 39 entries,
// BiCGSTAB, 4800 rows x 8 sets: 36 us an iteration with one, 28 with four).
// Lanes add up by warp shuffles, so only rows shared by lanes need a power of
// two of threads (18.7 k rows x 5 sets take 40.9 us a CG iteration with 8 threads
// to a row, 28.1 with 5), and on systems that fill the chip set counts that are
// none take one thread to a row and set.
static void product(symgb_solver_t s, const double* z, const double* w, double* y, double* d1, double* d2, double* zero,
                    double* zero2, cudaStream_t st) {
    unsigned width = 1;
    while (width < s->S) width *= 2;
    unsigned lanes = width == s->S ? std::max(1u, 8 / width) : 1;
    const std::uint64_t room = (std::uint64_t)s->smCount * 1024;
    const bool wide = width * lanes <= 32 && s->n * width * lanes <= room;
    while (wide && width * lanes < 32 && s->n * width * lanes * 2 <= room) lanes *= 2;
    if (lanes == 1 || !wide) width = s->S;
    auto launch = [&](auto fn) {
        launchStep(fn, s->blocks(s->n, wide ? 1024 : 2048, width, lanes), s->threads, s->sharedBytes(), st,
                   s->rowPtr.ptr, s->entry.ptr, s->vals.ptr, z, s->n, s->S, width, lanes, w, y, d1, d2, zero, zero2);
    };
    s->shared ? (wide ? launch(spmv<true, true>) : launch(spmv<true, false>))
              : (wide ? launch(spmv<false, true>) : launch(spmv<false, false>));
}

// Largest |r| / |b| of the S systems from their squares; infinity where one is
// not finite: NaN or Inf in the data, squares beyond the double range, or a
// breakdown, none of which an iteration comes back from.  `open`: some other
// system has not reached `tol`.
static double worstResidual(const double* rr, const double* bb, unsigned S, double tol, bool* open) {
    double worst = 0.0;
    *open = false;
    for (unsigned k = 0; k < S; ++k) {
        const double rel = rr[k] == 0.0 ? 0.0 : std::sqrt(rr[k] / bb[k]);
        if (!std::isfinite(rel) || !std::isfinite(bb[k])) {
            worst = std::numeric_limits<double>::infinity();
            continue;
        }
        worst = std::max(worst, rel);
        *open |= !(rel <= tol);
    }
    return worst;
}

int symgb_solver_multiply(symgb_solver_t s, const double* values, const double* p_dev, double* q_dev, void* stream) {
    using symgb::engine::setLastError;
    if (!s || !values || !p_dev || !q_dev) return setLastError(SYMGB_ERR_ARGUMENT, "solver: null argument");
    cudaStream_t st = (cudaStream_t)stream;
    const std::uint64_t work = s->n * s->S;
    if (int e = place(s, values, st)) return e;
    // p_dev and q_dev are [set][row]; the same transpose kernel with the roles
    // of rows and sets swapped gives the [row][set] copy of p.
    transposeSets<<<blocksFor(work), kThreads, 0, st>>>(p_dev, s->S, (unsigned)s->n, s->p.ptr);
    cudaMemsetAsync(s->scalars.ptr, 0, 8 * s->S * sizeof(double), st);
    product(s, s->p.ptr, s->p.ptr, s->q.ptr, s->scalars.ptr, nullptr, nullptr, nullptr, st);
    transposeSets<<<blocksFor(work), kThreads, 0, st>>>(s->q.ptr, s->n, s->S, q_dev);
    if (cudaStreamSynchronize(st) != cudaSuccess || cudaGetLastError() != cudaSuccess)
        return setLastError(SYMGB_ERR_CUDA, "solver: multiply failed");
    return SYMGB_OK;
}

static int solveCg(symgb_solver_t s, const double* values, const double* b_dev, double* x_dev, double tol, int max_iter,
                   void* stream, int* iterations, double* max_rel_residual) {
    using symgb::engine::setLastError;
    if (!s || !values || !b_dev || !x_dev || max_iter < 0) return setLastError(SYMGB_ERR_ARGUMENT, "solver: bad argument");
    cudaStream_t st = (cudaStream_t)stream;
    const unsigned S = s->S;
    const std::uint64_t work = s->n * S;
    // scalars: rz[2][S] (by iteration parity), pq[S], rr[S], bb[S]
    double* rz = s->scalars.ptr;
    double* pq = rz + 2 * S;
    double* rr = pq + S;
    double* bb = rr + S;
    const unsigned grid = s->vectorBlocks(s->n), block = s->threads;
    const std::size_t smem = s->sharedBytes();
    if (int e = place(s, values, st)) return e;
    cudaMemsetAsync(s->scalars.ptr, 0, 8 * (std::size_t)S * sizeof(double), st);
    cgStart<<<grid, block, smem, st>>>(b_dev, s->vals.ptr, s->diagPos.ptr, s->n, S, s->x.ptr, s->r.ptr, s->p.ptr,
                                       s->invDiag.ptr, rz, bb);
    int it = 0;
    double worst = 0.0;
    std::vector<double> bbHost(S);
    bool haveBb = false;
    while (it < max_iter) {
        const int count = std::min(kCheck, max_iter - it);
        for (int k = 0; k < count; ++k, ++it) {
            double* rzOld = rz + (it & 1) * S;
            double* rzNew = rz + ((it + 1) & 1) * S;
            product(s, s->p.ptr, s->p.ptr, s->q.ptr, pq, nullptr, rzNew, rr, st);
            launchStep(cgUpdate, grid, block, smem, st, s->p.ptr, s->q.ptr, s->invDiag.ptr, s->n, S, rzOld, pq, s->x.ptr,
                       s->r.ptr, rzNew, rr);
            launchStep(cgDirection, grid, block, smem, st, s->r.ptr, s->invDiag.ptr, s->n, S, rzOld, rzNew, s->p.ptr, pq);
        }
        if (!haveBb) {
            cudaMemcpyAsync(bbHost.data(), bb, S * sizeof(double), cudaMemcpyDeviceToHost, st);
            haveBb = true;
        }
        cudaMemcpyAsync(s->hostScalars, rr, S * sizeof(double), cudaMemcpyDeviceToHost, st);
        if (cudaStreamSynchronize(st) != cudaSuccess) return setLastError(SYMGB_ERR_CUDA, "solver: solve failed");
        bool open;
        worst = worstResidual(s->hostScalars, bbHost.data(), S, tol, &open);
        if (!open) break;
    }
    transposeSets<<<blocksFor(work), kThreads, 0, st>>>(s->x.ptr, s->n, S, x_dev);
    if (cudaStreamSynchronize(st) != cudaSuccess || cudaGetLastError() != cudaSuccess)
        return setLastError(SYMGB_ERR_CUDA, "solver: solve failed");
    if (iterations) *iterations = it;
    if (max_rel_residual) *max_rel_residual = max_iter ? worst : 1.0;
    return SYMGB_OK;
}

static int solveBicgstab(symgb_solver_t s, const double* values, const double* b_dev, double* x_dev, double tol,
                         int max_iter, void* stream, int* iterations, double* max_rel_residual) {
    using symgb::engine::setLastError;
    cudaStream_t st = (cudaStream_t)stream;
    const unsigned S = s->S;
    const std::uint64_t work = s->n * S;
    if (!s->rhat.ptr && (s->rhat.alloc(work) || s->v.alloc(work) || s->ph.alloc(work) || s->sv.alloc(work) ||
                         s->sh.alloc(work) || s->t.alloc(work)))
        return setLastError(SYMGB_ERR_NOMEM, "solver: device allocation failed");
    double* R = s->scalars.ptr;  // rho[2][S] by iteration parity
    double* rv = R + 2 * S;      // rv, ts, tt, rr contiguous
    double* ts = rv + S;
    double* tt = ts + S;
    double* rr = tt + S;
    double* bb = rr + S;
    double* alpha = bb + S;
    double* omega = alpha + S;
    const unsigned grid = s->vectorBlocks(s->n), block = s->threads;
    const std::size_t smem = s->sharedBytes();
    if (int e = place(s, values, st)) return e;
    cudaMemsetAsync(s->scalars.ptr, 0, 16 * (std::size_t)S * sizeof(double), st);
    bStart<<<grid, block, smem, st>>>(b_dev, s->vals.ptr, s->diagPos.ptr, s->n, S, s->x.ptr, s->r.ptr, s->rhat.ptr,
                                      s->p.ptr, s->v.ptr, s->invDiag.ptr, R, R + S, alpha, omega, bb);
    const int B = s->block;
    if (B > 1) blockInvertLaunch(B, s->vals.ptr, s->blockPos.ptr, s->n / B, S, s->blockInv.ptr, st);
    const double* inv = B > 1 ? s->blockInv.ptr : s->invDiag.ptr;
    const std::uint64_t nb = s->n / B, stride = B > 1 ? s->blockStride : 1;
    const unsigned nodeGrid = s->vectorBlocks(nb);
    int it = 0;
    double worst = 0.0;
    std::vector<double> bbHost(S);
    bool haveBb = false;
    while (it < max_iter) {
        const int count = std::min(kCheck, max_iter - it);
        for (int k = 0; k < count; ++k, ++it) {
            double* rho = R + (it & 1) * S;
            double* rhoOther = R + ((it + 1) & 1) * S;  // the previous one, then the next one's sum
            auto direction = [&](auto fn) {
                launchStep(fn, nodeGrid, block, smem, st, s->r.ptr, s->v.ptr, inv, nb, stride, S, rho, rhoOther, alpha,
                           omega, s->p.ptr, s->ph.ptr, rv);
            };
            auto half = [&](auto fn) {
                launchStep(fn, nodeGrid, block, smem, st, s->r.ptr, s->v.ptr, inv, nb, stride, S, rho, rv, alpha, s->sv.ptr,
                           s->sh.ptr);
            };
            B == 1 ? direction(bDirection<1>) : B == 2 ? direction(bDirection<2>) : B == 3 ? direction(bDirection<3>)
                                                                                        : direction(bDirection<4>);
            product(s, s->ph.ptr, s->rhat.ptr, s->v.ptr, rv, nullptr, rhoOther, nullptr, st);
            B == 1 ? half(bHalf<1>) : B == 2 ? half(bHalf<2>) : B == 3 ? half(bHalf<3>) : half(bHalf<4>);
            product(s, s->sh.ptr, s->sv.ptr, s->t.ptr, ts, tt, nullptr, nullptr, st);
            launchStep(bFinishStep, grid, block, smem, st, s->ph.ptr, s->sh.ptr, s->sv.ptr, s->t.ptr, s->rhat.ptr, s->n,
                       S, alpha, ts, tt, omega, s->x.ptr, s->r.ptr, rhoOther, rr);
        }
        if (!haveBb) {
            cudaMemcpyAsync(bbHost.data(), bb, S * sizeof(double), cudaMemcpyDeviceToHost, st);
            haveBb = true;
        }
        cudaMemcpyAsync(s->hostScalars, rr, S * sizeof(double), cudaMemcpyDeviceToHost, st);
        if (cudaStreamSynchronize(st) != cudaSuccess) return setLastError(SYMGB_ERR_CUDA, "solver: solve failed");
        bool open;
        worst = worstResidual(s->hostScalars, bbHost.data(), S, tol, &open);
        if (!open) break;
    }
    transposeSets<<<blocksFor(work), kThreads, 0, st>>>(s->x.ptr, s->n, S, x_dev);
    if (cudaStreamSynchronize(st) != cudaSuccess || cudaGetLastError() != cudaSuccess)
        return setLastError(SYMGB_ERR_CUDA, "solver: solve failed");
    if (iterations) *iterations = it;
    if (max_rel_residual) *max_rel_residual = max_iter ? worst : 1.0;
    return SYMGB_OK;
}

int symgb_solver_solve(symgb_solver_t s, int method, const double* values, const double* b, double* x, double tol,
                       int max_iter, void* stream, int* iterations, double* max_rel_residual) {
    using symgb::engine::setLastError;
    if (!s || !values || !b || !x || max_iter < 0) return setLastError(SYMGB_ERR_ARGUMENT, "solver: bad argument");
    if (method == SYMGB_SOLVER_CG) return solveCg(s, values, b, x, tol, max_iter, stream, iterations, max_rel_residual);
    if (method == SYMGB_SOLVER_BICGSTAB)
        return solveBicgstab(s, values, b, x, tol, max_iter, stream, iterations, max_rel_residual);
    return setLastError(SYMGB_ERR_ARGUMENT, "solver: unknown method");
}

void symgb_solver_destroy(symgb_solver_t s) { delete s; }

}  // extern "C"
