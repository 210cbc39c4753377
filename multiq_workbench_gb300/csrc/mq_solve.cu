// Device Laplace solver: the host solver of mq_grid.cpp (conjugate gradients preconditioned by a
// symmetric geometric V-cycle with red-black Gauss-Seidel smoothing, stopping on the scaled
// max-norm residual) run on the GPU with the same arithmetic in the same order, so the two give
// bit-identical potentials: every node update is the host's expression (this unit is compiled
// without FMA contraction), a colour's nodes are independent within a half sweep, and the dot
// products are summed row by row, plane by plane, exactly as the host sums them. The electrodes of a
// channel geometry and its E field are formed here too, with the host's expressions.
//
// Replaces the set-up step before the path (fieldsolve's solve, simulation/fieldsolve/src/lib.rs:164,
// as restated by mq_laplace_solve) where grids of 10^7-10^8 nodes make the host solve the cost.
//
// What bounds it: GB300's FP64 pipe (one warp instruction per 19 cycles and SM) and the traffic of the
// finest level, which just fits L2; below it launches and chains of additions. So what need not be FP64
// arithmetic is not: the division by 6 and the scaling by powers of two of restriction and prolongation
// run on the integer pipe with the same roundings, sums over a zero iterate are not formed, and the
// prolongation leaves out the colour that the next half sweep overwrites. The ordered dot products are
// chains of additions: 32 rows are summed side by side from shared memory while other warps form the
// next terms. The host sets nothing up: mask, coarse masks and initial iterate are formed here, and its
// part of an iteration is one synchronisation.
// Measured on the 0.100 mm channel (160 x 160 x 242, 10 iterations), per basis, before -> now: kernels 24 -> 9.9 ms
// (half sweeps 9.4 -> 3.6, of which one of the finest level is 22 us; prolongation 2.7 -> 0.5; ordered sums and S p
// 3.7 -> 2.0; coarsest level 2.1 -> 0.9 with two levels more in the same launch; restriction 2.0 -> 0.7; residuals
// 1.2 -> 0.5), the whole call 55 -> 11.5 ms, of which 30 were the host's part.
#include <sys/mman.h>
#include <unistd.h>

#include <chrono>
#include <cmath>
#include <cstring>
#include <functional>
#include <thread>
#include <vector>

#include "mq_chan_geom.h"
#include "mq_check.h"
#include "mq_grid.h"
#include "mq_levels.h"
#include "mq_phys.h"
#include "mq_solve_dev.h"

namespace {

constexpr int kT = 256;

struct DLevel {
    int nx, ny, nz;
    uint8_t* fix;
    double *u, *rhs, *r;
    uint32_t* list[2];   // free nodes by colour, or null (k_list)
    uint32_t cnt[2];
    size_t n() const { return (size_t)nx * ny * nz; }
};

// scalars of the iteration, on the device
struct Scal {
    double rz, pq, alpha, beta;
    unsigned long long rmax;   // bits of max |r|
    unsigned int done;         // planes summed so far
};

// x / 6, correctly rounded, on the integer pipe: with m the 53-bit significand, m / 3 scaled to 53 bits is
// floor((m 2^s + 1) / 3) (a remainder of 1 rounds down, 2 up, and no quotient by 3 is a tie), s = 1 for
// m >= 1.5 2^52 and 2 below. Zeros keep their sign; values near the ends of the range, infinities and
// NaN take the division.
__device__ __forceinline__ double div6(double x) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(x);
    const unsigned e = (unsigned)(b >> 52) & 0x7ffu;
    if (e - 4u >= 2043u) return (b << 1) == 0ull ? x : x / 6.0;
    const unsigned long long m = (b & 0xfffffffffffffull) | 0x10000000000000ull;
    const int s = m >= 0x18000000000000ull ? 1 : 2;
    const unsigned long long q = __umul64hi((m << s) + 1ull, 0xaaaaaaaaaaaaaaabull) >> 1;   // [2^52, 2^53)
    return __longlong_as_double((long long)((b & 0x8000000000000000ull) + ((unsigned long long)(e - 2u - (unsigned)s) << 52) + q));
}

// 2^-k
__device__ __forceinline__ double pow2m(int k) { return __hiloint2double(0x3ff00000 - (k << 20), 0); }

__device__ __forceinline__ bool is_zero(double x) { return ((__double2hiint(x) << 1) | __double2loint(x)) == 0; }

// x 2^-k, on the integer pipe but near the ends of the range
__device__ __forceinline__ double down2(double x, int k) {
    const int hi = __double2hiint(x), e = hi & 0x7ff00000, d = k << 20;
    if (e > d && e != 0x7ff00000) return __hiloint2double(hi - d, __double2loint(x));
    return is_zero(x) ? x : x * pow2m(k);
}

// 0.0 + p: p, but +0 for -0
__device__ __forceinline__ double plus_zero(double p) {
    return __double_as_longlong(p) == (long long)0x8000000000000000ULL ? 0.0 : p;
}

// plane of a block in a grid of plane_blocks()
__device__ __forceinline__ int block_plane() { return (int)(blockIdx.y + gridDim.y * blockIdx.z); }

// ---------------------------------------------------------------- smoothing
// node of thread t of a colour's half sweep in plane k; false where there is none
__device__ __forceinline__ bool colour_node(unsigned t, int k, int col, int nx, int ny, size_t& q, int& i, int& j) {
    const unsigned hx = (unsigned)(nx - 1) / 2u;
    j = 1 + (int)(t / hx);
    i = 1 + ((1 + j + k + col) & 1) + 2 * (int)(t % hx);
    q = (size_t)i + (size_t)nx * ((size_t)j + (size_t)ny * (size_t)k);
    return j < ny - 1 && i <= nx - 2;
}
__device__ __forceinline__ bool colour_node(unsigned t, int k, int col, int nx, int ny, size_t& q) {
    int i, j;
    return colour_node(t, k, col, nx, ny, q, i, j);
}

// The free nodes of a colour, in runs of up to 256 neighbours. Half of a channel's nodes lie in electrodes, and its rows
// cross them: warps over all nodes of a colour have 60 in 100 lanes at work, warps over this list all of them,
// and the FP64 pipe's time goes by warps (half sweep of the finest level of the 0.100 mm channel 35 -> 22 us, the list once a
// solve 20 us).
__global__ void __launch_bounds__(kT) k_list(const uint8_t* __restrict__ fix, int nx, int ny, int nz, int col, uint32_t* __restrict__ list,
                                             [[maybe_unused]] size_t room, uint32_t* __restrict__ cnt) {
    __shared__ uint32_t warp_n[kT / 32], base;
    const int k = 1 + block_plane();
    size_t q = 0;
    const bool f = k <= nz - 2 && colour_node(blockIdx.x * kT + threadIdx.x, k, col, nx, ny, q) && !fix[q];
    const unsigned b = __ballot_sync(0xffffffffu, f), lane = threadIdx.x & 31u, w = threadIdx.x >> 5;
    if (lane == 0) warp_n[w] = (uint32_t)__popc(b);
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t n = 0;
        for (int x = 0; x < kT / 32; ++x) { const uint32_t m = warp_n[x]; warp_n[x] = n; n += m; }
        base = n ? atomicAdd(cnt, n) : 0u;
    }
    __syncthreads();
    if (f) list[MQ_CHK(base + warp_n[w] + (uint32_t)__popc(b & ((1u << lane) - 1u)), room, MQ_SITE_SOLVE_LIST)] = (uint32_t)q;
}
// node of this thread: the list's, or where there is none (grids of 2^32 nodes and more) the colour's free nodes in turn
__device__ __forceinline__ bool free_node(const uint32_t* __restrict__ list, uint32_t cnt, const uint8_t* __restrict__ fix, int col, int nx,
                                          int ny, int nz, size_t& q) {
    const unsigned t = blockIdx.x * kT + threadIdx.x;
    if (list) {
        if (t >= cnt) return false;
        q = MQ_CHK(list[t], (size_t)nx * ny * nz, MQ_SITE_SOLVE_NODE);
        return true;
    }
    const int k = 1 + block_plane();
    return k <= nz - 2 && colour_node(t, k, col, nx, ny, q) && !fix[q];
}

// RES: also the residual at the nodes updated, whose neighbours stay as they are here
template <bool RES>
__global__ void __launch_bounds__(kT) k_gs(double* __restrict__ u, const double* __restrict__ rhs, const uint8_t* __restrict__ fix,
                                           double* __restrict__ r, int nx, int ny, int nz, int col, const uint32_t* __restrict__ list,
                                           uint32_t cnt) {
    size_t q;
    if (!free_node(list, cnt, fix, col, nx, ny, nz, q)) return;
    const size_t sy = nx, sz = (size_t)nx * ny;
    const double s = u[q - 1] + u[q + 1] + u[q - sy] + u[q + sy] + u[q - sz] + u[q + sz];
    const double a = rhs[q] + s, v = div6(a);
    u[q] = v;
    if (RES) r[q] = a - 6.0 * v;
}

// the first half sweep (colour 0) on u = 0: the neighbours' sum is 0. Colour 1's nodes are not read before they are
// set anew, and fixed ones are 0 from the start.
__global__ void __launch_bounds__(kT) k_gs_first(double* __restrict__ u, const double* __restrict__ rhs, const uint8_t* __restrict__ fix,
                                                 int nx, int ny, int nz, const uint32_t* __restrict__ list, uint32_t cnt) {
    size_t q;
    if (free_node(list, cnt, fix, 0, nx, ny, nz, q)) u[q] = div6(plus_zero(rhs[q]));
}

// A coarsest level too large for k_bottom (a long thin grid's, the hierarchy ends below 5 nodes on one
// axis): sweeps x (red, black, black, red) from u = 0 in one block. A half sweep right after one of its own
// colour changes nothing and is left out.
__global__ void __launch_bounds__(1024) k_coarse(double* u, const double* rhs, const uint8_t* fix, int nx, int ny, int nz, int sweeps) {
    const long long n = (long long)nx * ny * nz, sy = nx, sz = (long long)nx * ny;
    for (long long q = threadIdx.x; q < n; q += blockDim.x) u[q] = 0.0;
    __syncthreads();
    const int hx = (nx - 1) / 2;
    const long long total = (long long)hx * (ny - 2) * (nz - 2);
    for (int h = 0; h <= 2 * sweeps; ++h) {
        for (long long t = threadIdx.x; t < total; t += blockDim.x) {
            const int m = (int)(t % hx);
            const long long row = t / hx;
            const int j = 1 + (int)(row % (ny - 2)), k = 1 + (int)(row / (ny - 2));
            const int i = 1 + ((1 + j + k + h) & 1) + 2 * m;   // colour h & 1
            if (i > nx - 2) continue;
            const long long q = i + sy * j + sz * k;
            if (fix[q]) continue;
            const double v = u[q - 1] + u[q + 1] + u[q - sy] + u[q + sy] + u[q - sz] + u[q + sz];
            u[q] = div6(rhs[q] + v);
        }
        __syncthreads();
    }
}

// ---------------------------------------------------------------- grid transfer
// residual at the free nodes of colour 0 (k_gs<true> has left colour 1's; it stays 0 at fixed nodes)
__global__ void __launch_bounds__(kT) k_residual(const double* __restrict__ u, const double* __restrict__ rhs,
                                                 const uint8_t* __restrict__ fix, double* __restrict__ r, int nx, int ny, int nz,
                                                 const uint32_t* __restrict__ list, uint32_t cnt) {
    size_t q;
    if (!free_node(list, cnt, fix, 0, nx, ny, nz, q)) return;
    const size_t sy = nx, sz = (size_t)nx * ny;
    const double s = u[q - 1] + u[q + 1] + u[q - sy] + u[q + sy] + u[q - sz] + u[q + sz];
    r[q] = rhs[q] + s - 6.0 * u[q];
}

// half the full weighting around the fine node f: every weight is a power of two. The 27 fine nodes of a free coarse node lie in
// the fine grid (coarse faces and nodes beyond it are fixed).
template <class I>
__device__ __forceinline__ double restrict_node(const double* f, I sy, I sz) {
    double s = 0.0;
#pragma unroll
    for (int dk = -1; dk <= 1; ++dk)
#pragma unroll
        for (int dj = -1; dj <= 1; ++dj)
#pragma unroll
            for (int di = -1; di <= 1; ++di) {
                const int k = (dk != 0) + (dj != 0) + (di != 0);
                const double v = f[di + sy * dj + sz * dk];
                s += k ? down2(v, k) : v;
            }
    return down2(s, 1);
}
__global__ void __launch_bounds__(kT) k_restrict(const double* __restrict__ fr, int fnx, int fny, double* __restrict__ crhs,
                                                 const uint8_t* __restrict__ cfix, int cnx, int cny, int cnz,
                                                 const uint32_t* __restrict__ l0, uint32_t n0, const uint32_t* __restrict__ l1, uint32_t n1) {
    const unsigned t = blockIdx.x * kT + threadIdx.x, n = (unsigned)cnx * (unsigned)cny;
    unsigned I, J, K;
    size_t qc;
    if (l0) {   // free nodes only: nothing reads the others' right-hand side
        if (t >= n0 + n1) return;
        const unsigned x = (unsigned)MQ_CHK(t < n0 ? l0[t] : l1[t - n0], (size_t)n * cnz, MQ_SITE_SOLVE_NODE), y = x / (unsigned)cnx;
        I = x % (unsigned)cnx; J = y % (unsigned)cny; K = y / (unsigned)cny;
        qc = x;
    } else {
        K = (unsigned)block_plane();
        if (t >= n || K >= (unsigned)cnz) return;
        I = t % (unsigned)cnx; J = t / (unsigned)cnx;
        qc = (size_t)t + (size_t)n * K;
        if (cfix[qc]) { crhs[qc] = 0.0; return; }
    }
    const size_t sy = fnx, sz = (size_t)fnx * fny;
    crhs[qc] = restrict_node(fr + (size_t)(2 * I) + sy * (size_t)(2 * J) + sz * (size_t)(2 * K), (ptrdiff_t)sy, (ptrdiff_t)sz);
}

// P cu at a fine node with odd coordinates oi, oj, ok above the coarse node c. Its corners all have the weight
// 2^-(odd coordinates). It multiplies their sum, which rounds as the sum of the weighted corners does,
// unless a corner is so small that its product is rounded, or so large that the sum overflows: then it
// multiplies them one by one.
template <class I>
__device__ __forceinline__ double prolong_node(const double* c, I sy, I sz, bool oi, bool oj, bool ok) {
    const int w = (int)oi + (int)oj + (int)ok;
    double v[8];
    bool odd = false;
#pragma unroll
    for (unsigned x = 0; x < 8; ++x) {
        const bool use = (!(x & 1u) || oi) && (!(x & 2u) || oj) && (!(x & 4u) || ok);
        v[x] = use ? c[(x & 1u ? (I)1 : (I)0) + (x & 2u ? sy : (I)0) + (x & 4u ? sz : (I)0)] : 0.0;
        odd |= ((__double2hiint(v[x]) >> 20 & 0x7ff) - 4u) >= 2036u && !is_zero(v[x]);
    }
    if (odd) {
#pragma unroll
        for (int x = 0; x < 8; ++x) v[x] *= pow2m(w);
    }
    double s = plus_zero(v[0]);
    if (oi) s += v[1];
    if (oj) {
        s += v[2];
        if (oi) s += v[3];
    }
    if (ok) {
        s += v[4];
        if (oi) s += v[5];
        if (oj) {
            s += v[6];
            if (oi) s += v[7];
        }
    }
    return odd ? s : down2(s, w);
}

// fu += P cu at colour 0: the half sweep over colour 1 that follows reads no value of its own colour
__global__ void __launch_bounds__(kT) k_prolong(const double* __restrict__ cu, int cnx, int cny, double* __restrict__ fu,
                                                const uint8_t* __restrict__ ffix, int fnx, int fny, int fnz,
                                                const uint32_t* __restrict__ list, uint32_t cnt) {
    size_t q;
    if (!free_node(list, cnt, ffix, 0, fnx, fny, fnz, q)) return;
    int i, j, k;
    if (list) {
        const unsigned x = (unsigned)q, y = x / (unsigned)fnx;
        i = (int)(x % (unsigned)fnx); j = (int)(y % (unsigned)fny); k = (int)(y / (unsigned)fny);
    } else {
        i = (int)(q % (size_t)fnx); j = (int)(q / (size_t)fnx % (size_t)fny); k = (int)(q / ((size_t)fnx * fny));
    }
    const size_t sy = cnx, sz = (size_t)cnx * cny;
    fu[q] += prolong_node(cu + (size_t)(i / 2) + sy * (size_t)(j / 2) + sz * (size_t)(k / 2), sy, sz, i & 1, j & 1, k & 1);
}

// ---------------------------------------------------------------- the small levels in one block
// The V-cycle below a level of a few thousand nodes, in shared memory: as launches of their own its half
// sweeps are 3.5 to 4 us each, whatever their size; three levels and the coarsest one's 121 half sweeps are 79 us
// here (a level of 2600 nodes costs about what its launches do, so the line lies there). The coarsest level's half
// sweeps are a chain of additions and run in one warp if they fit.
constexpr int kBottomNodes = 2600, kBottomLevels = 8;
struct Bottom {
    int levels, nx[kBottomLevels], ny[kBottomLevels], nz[kBottomLevels];
    const uint8_t* fix[kBottomLevels];
};
struct SLevel {
    int nx, ny, nz;
    double *u, *rhs, *r;
    uint8_t* fix;
};

// node of slot t of a colour's half sweep, or -1
__device__ __forceinline__ int slot(const SLevel& v, int t, int col) {
    const int hx = (v.nx - 1) / 2, m = t % hx, row = t / hx, j = 1 + row % (v.ny - 2), k = 1 + row / (v.ny - 2);
    const int i = 1 + ((1 + j + k + col) & 1) + 2 * m, q = i + v.nx * (j + v.ny * k);
    return i > v.nx - 2 || v.fix[q] ? -1 : q;
}
__device__ __forceinline__ void relax(const SLevel& v, int q, double rhs) {
    const int sy = v.nx, sz = v.nx * v.ny;
    const double s = v.u[q - 1] + v.u[q + 1] + v.u[q - sy] + v.u[q + sy] + v.u[q - sz] + v.u[q + sz];
    v.u[q] = div6(rhs + s);
}
__device__ __forceinline__ int slots(const SLevel& v) { return (v.nx - 1) / 2 * (v.ny - 2) * (v.nz - 2); }
__device__ void half_sweep(const SLevel& v, int col) {
    const int total = slots(v);
    for (int t = threadIdx.x; t < total; t += blockDim.x) {
        const int q = slot(v, t, col);
        if (q >= 0) relax(v, q, v.rhs[q]);
    }
    __syncthreads();
}

__global__ void __launch_bounds__(1024) k_bottom(const __grid_constant__ Bottom B, const double* __restrict__ grhs, double* __restrict__ gu,
                                                 int sweeps) {
    extern __shared__ double mem[];
    SLevel V[kBottomLevels];
    int nodes = 0;
#pragma unroll
    for (int l = 0; l < kBottomLevels; ++l)
        if (l < B.levels) nodes += B.nx[l] * B.ny[l] * B.nz[l];
    int off = 0;
#pragma unroll
    for (int l = 0; l < kBottomLevels; ++l) {
        if (l >= B.levels) break;
        SLevel& v = V[l];
        v.nx = B.nx[l]; v.ny = B.ny[l]; v.nz = B.nz[l];
        v.u = mem + off; v.rhs = mem + nodes + off; v.r = mem + 2 * nodes + off;
        v.fix = reinterpret_cast<uint8_t*>(mem + 3 * nodes) + off;
        const int n = v.nx * v.ny * v.nz;
        for (int q = threadIdx.x; q < n; q += blockDim.x) {
            v.fix[q] = B.fix[l][q];
            if (l == 0) v.rhs[q] = grhs[q];
        }
        off += n;
    }
    __syncthreads();
    const int last = B.levels - 1;
    for (int l = 0; l < last; ++l) {
        const SLevel &v = V[l], &c = V[l + 1];
        const int n = v.nx * v.ny * v.nz, sy = v.nx, sz = v.nx * v.ny;
        for (int q = threadIdx.x; q < n; q += blockDim.x) {
            const int i = q % v.nx, j = q / v.nx % v.ny, k = q / sz;
            v.u[q] = ((i + j + k) & 1) == 0 && !v.fix[q] ? div6(plus_zero(v.rhs[q])) : 0.0;
        }
        __syncthreads();
        half_sweep(v, 1);
        half_sweep(v, 0);
        half_sweep(v, 1);
        for (int q = threadIdx.x; q < n; q += blockDim.x) {
            double r = 0.0;
            if (!v.fix[q]) {
                const double s = v.u[q - 1] + v.u[q + 1] + v.u[q - sy] + v.u[q + sy] + v.u[q - sz] + v.u[q + sz];
                r = v.rhs[q] + s - 6.0 * v.u[q];
            }
            v.r[q] = r;
        }
        __syncthreads();
        const int nc = c.nx * c.ny * c.nz, cz = c.nx * c.ny;
        for (int q = threadIdx.x; q < nc; q += blockDim.x) {
            const int i = q % c.nx, j = q / c.nx % c.ny, k = q / cz;
            c.rhs[q] = c.fix[q] ? 0.0 : restrict_node(v.r + 2 * i + sy * (2 * j) + sz * (2 * k), sy, sz);
        }
        __syncthreads();
    }
    {
        const SLevel& v = V[last];
        const int n = v.nx * v.ny * v.nz, total = slots(v);
        for (int q = threadIdx.x; q < n; q += blockDim.x) v.u[q] = 0.0;
        __syncthreads();
        if (total > 32) {
            for (int h = 0; h <= 2 * sweeps; ++h) half_sweep(v, h & 1);
        } else if (threadIdx.x < 32) {
            const int t = (int)threadIdx.x, q0 = t < total ? slot(v, t, 0) : -1, q1 = t < total ? slot(v, t, 1) : -1;
            const double r0 = q0 >= 0 ? v.rhs[q0] : 0.0, r1 = q1 >= 0 ? v.rhs[q1] : 0.0;
            if (q0 >= 0) relax(v, q0, r0);
            __syncwarp();
            for (int s = 0; s < sweeps; ++s) {
                if (q1 >= 0) relax(v, q1, r1);
                __syncwarp();
                if (q0 >= 0) relax(v, q0, r0);
                __syncwarp();
            }
        }
        __syncthreads();
    }
    for (int l = last - 1; l >= 0; --l) {
        const SLevel &v = V[l], &c = V[l + 1];
        const int total = slots(v), sy = v.nx, sz = v.nx * v.ny, cy = c.nx, cz = c.nx * c.ny;
        for (int t = threadIdx.x; t < total; t += blockDim.x) {
            const int q = slot(v, t, 0);
            if (q < 0) continue;
            const int i = q % sy, j = q / sy % v.ny, k = q / sz;
            v.u[q] += prolong_node(c.u + i / 2 + cy * (j / 2) + cz * (k / 2), cy, cz, i & 1, j & 1, k & 1);
        }
        __syncthreads();
        for (int s = 0; s < 2; ++s) {
            half_sweep(v, 1);
            half_sweep(v, 0);
        }
    }
    const int n0 = V[0].nx * V[0].ny * V[0].nz;
    for (int q = threadIdx.x; q < n0; q += blockDim.x) gu[q] = V[0].u[q];
}

// ---------------------------------------------------------------- reductions
// max of non-negative doubles by their bits (NaN left out), one atomic per block
__device__ __forceinline__ unsigned long long abs_bits(double v) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(v) & 0x7fffffffffffffffull;
    return b > 0x7ff0000000000000ull ? 0ull : b;
}
__device__ __forceinline__ void block_max(unsigned long long m, unsigned long long* out) {
    __shared__ unsigned long long w[kT / 32];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long x = __shfl_down_sync(0xffffffffu, m, o);
        m = x > m ? x : m;
    }
    if ((threadIdx.x & 31) == 0) w[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int k = 1; k < kT / 32; ++k) m = w[k] > m ? w[k] : m;
        if (m) atomicMax(out, m);
    }
}

// r = S-residual of phi at free nodes (sum of neighbours - 6 phi), 0 at fixed; max |r|
__global__ void __launch_bounds__(kT) k_true_residual(const double* __restrict__ phi, const uint8_t* __restrict__ fix,
                                                      double* __restrict__ r, int nx, int ny, size_t n, Scal* __restrict__ sc) {
    unsigned long long m = 0;
    const size_t sy = nx, sz = (size_t)nx * ny;
    for (size_t q = (size_t)blockIdx.x * kT + threadIdx.x; q < n; q += (size_t)gridDim.x * kT) {
        double v = 0.0;
        if (!fix[q]) {
            const double s = phi[q - 1] + phi[q + 1] + phi[q - sy] + phi[q + sy] + phi[q - sz] + phi[q + sz];
            v = s - 6.0 * phi[q];
        }
        r[q] = v;
        const unsigned long long b = abs_bits(v);
        m = b > m ? b : m;
    }
    block_max(m, &sc->rmax);
}

// Row sums in i order. STENCIL: q = S p at free nodes (0 at fixed), terms p q; else terms a b. Warp 0 adds up 32
// rows, one per lane, while the other eight warps form the next 32 columns' terms in shared memory.
constexpr int kRows = 32;
template <bool STENCIL>
__global__ void __launch_bounds__(kT + 32) k_rows(const double* __restrict__ a, const double* __restrict__ b,
                                                  const uint8_t* __restrict__ fix, double* __restrict__ qv, int nx, int ny, size_t rows,
                                                  double* __restrict__ rowsum) {
    __shared__ double tile[2][kRows][33];
    const size_t row0 = (size_t)blockIdx.x * kRows;
    const int lane = threadIdx.x & 31, w = (int)(threadIdx.x >> 5) - 1;
    const size_t sy = nx, sz = (size_t)nx * ny;
    const int chunks = (nx + 31) / 32;
    double s = 0.0;
    for (int c = 0; c <= chunks; ++c) {
        if (w >= 0 && c < chunks) {
            const int i = 32 * c + lane;
#pragma unroll
            for (int x = 0; x < kRows / 8; ++x) {
                const int lr = w * (kRows / 8) + x;
                double term = 0.0;
                if (row0 + lr < rows && i < nx) {
                    const size_t q = (row0 + lr) * sy + (size_t)i;
                    if (STENCIL) {
                        double v = 0.0;
                        if (!fix[q]) {
                            const double nb = a[q - 1] + a[q + 1] + a[q - sy] + a[q + sy] + a[q - sz] + a[q + sz];
                            v = 6.0 * a[q] - nb;
                            term = a[q] * v;
                        }
                        qv[q] = v;
                    } else {
                        term = a[q] * b[q];
                    }
                }
                tile[c & 1][lr][lane] = term;
            }
        }
        if (w < 0 && c > 0) {
            const int m = nx - 32 * (c - 1);
            if (m >= 32) {
#pragma unroll
                for (int x = 0; x < 32; ++x) s += tile[(c - 1) & 1][lane][x];
            } else {
                for (int x = 0; x < m; ++x) s += tile[(c - 1) & 1][lane][x];
            }
        }
        __syncthreads();
    }
    if (w < 0 && row0 + lane < rows) rowsum[row0 + lane] = s;
}

// ordered sum of n values by one warp (every lane has it)
__device__ __forceinline__ double ordered_sum(const double* v, int n, int lane) {
    double s = 0.0, next = lane < n ? __ldcg(v + lane) : 0.0;
    for (int c = 0; c < n; c += 32) {
        const double cur = next;
        next = c + 32 + lane < n ? __ldcg(v + c + 32 + lane) : 0.0;
        if (n - c >= 32) {
#pragma unroll
            for (int x = 0; x < 32; ++x) s += __shfl_sync(0xffffffffu, cur, x);
        } else {
            for (int x = 0; x < n - c; ++x) s += __shfl_sync(0xffffffffu, cur, x);
        }
    }
    return s;
}

// plane sums of the rows in j order (one warp per plane), then the planes in k order by the last of them, and the
// step's scalars: RZ0: r z of a new direction; ALPHA: p q and alpha = rz / pq; BETA: beta = rz' / rz
enum Sum { RZ0, ALPHA, BETA };
__global__ void __launch_bounds__(32) k_planes(const double* __restrict__ rowsum, int ny, double* plane, Scal* sc, Sum what) {
    const int lane = threadIdx.x;
    const double s = ordered_sum(rowsum + (size_t)blockIdx.x * ny, ny, lane);
    unsigned last = 0;
    if (lane == 0) {
        *(volatile double*)&plane[blockIdx.x] = s;
        __threadfence();
        last = atomicAdd(&sc->done, 1u) + 1u == gridDim.x;
    }
    if (!__shfl_sync(0xffffffffu, last, 0)) return;
    __threadfence();
    const double v = ordered_sum(plane, (int)gridDim.x, lane);
    if (lane == 0) {
        sc->done = 0;
        if (what == RZ0) sc->rz = v;
        else if (what == ALPHA) { sc->pq = v; sc->alpha = sc->rz / v; sc->rmax = 0; }
        else { sc->beta = v / sc->rz; sc->rz = v; }
    }
}

// phi += alpha p, r -= alpha q, max |r|; nothing if p q is not positive. p, q and r are 0 at fixed nodes, where only the
// first update (`all`) changes anything: a potential of -0 to +0 (70 -> 60 us; in the sums and the direction the look
// at the mask costs what it saves).
__global__ void __launch_bounds__(kT) k_cg_update(double* __restrict__ phi, double* __restrict__ r, const double* __restrict__ p,
                                                  const double* __restrict__ qv, const uint8_t* __restrict__ fix, size_t n, bool all,
                                                  Scal* __restrict__ sc) {
    if (!(sc->pq > 0)) return;
    const double alpha = sc->alpha;
    unsigned long long m = 0;
    for (size_t q = (size_t)blockIdx.x * kT + threadIdx.x; q < n; q += (size_t)gridDim.x * kT) {
        if (!all && fix[q]) continue;
        phi[q] += alpha * p[q];
        const double v = r[q] - alpha * qv[q];
        r[q] = v;
        const unsigned long long b = abs_bits(v);
        m = b > m ? b : m;
    }
    block_max(m, &sc->rmax);
}

// p = z + beta p
__global__ void __launch_bounds__(kT) k_cg_dir(double* __restrict__ p, const double* __restrict__ z, size_t n, const Scal* __restrict__ sc) {
    const size_t q = (size_t)blockIdx.x * kT + threadIdx.x;
    if (q < n) p[q] = z[q] + sc->beta * p[q];
}

// ---------------------------------------------------------------- the problem
// Dirichlet set and initial iterate as the host solver builds them, and max |fixed|
__global__ void __launch_bounds__(kT) k_problem(const uint8_t* __restrict__ mask, const double* __restrict__ fixed, double outer, int nx,
                                                int ny, int nz, uint8_t* __restrict__ fix, double* __restrict__ phi, Scal* __restrict__ sc) {
    const size_t n = (size_t)nx * ny * nz;
    unsigned long long m = 0;
    for (size_t q = (size_t)blockIdx.x * kT + threadIdx.x; q < n; q += (size_t)gridDim.x * kT) {
        const int i = (int)(q % (size_t)nx), j = (int)(q / (size_t)nx % (size_t)ny), k = (int)(q / ((size_t)nx * ny));
        const bool face = i == 0 || j == 0 || k == 0 || i == nx - 1 || j == ny - 1 || k == nz - 1;
        const bool solid = mask[q] != 0;
        const double f = solid ? fixed[q] : 0.0;
        fix[q] = solid || face ? 1 : 0;
        phi[q] = solid ? f : outer;
        const unsigned long long b = solid ? abs_bits(f) : 0ull;
        m = b > m ? b : m;
    }
    block_max(m, &sc->rmax);
}

// the same for a basis of a channel geometry: its electrodes are found here
__global__ void __launch_bounds__(kT) k_channel(const mq_geom g, const mqgeo::Layers L, int basis, double outer, int nx, int ny, int nz,
                                                uint8_t* __restrict__ mask, uint8_t* __restrict__ fix, double* __restrict__ phi,
                                                Scal* __restrict__ sc) {
    const size_t n = (size_t)nx * ny * nz;
    unsigned long long m = 0;
    for (size_t q = (size_t)blockIdx.x * kT + threadIdx.x; q < n; q += (size_t)gridDim.x * kT) {
        const int i = (int)(q % (size_t)nx), j = (int)(q / (size_t)nx % (size_t)ny), k = (int)(q / ((size_t)nx * ny));
        const bool face = i == 0 || j == 0 || k == 0 || i == nx - 1 || j == ny - 1 || k == nz - 1;
        const uint8_t e = mqgeo::classify(&g, L, i, j, k);
        const double f = e ? mqgeo::basis_value(basis, e, g.ac_mode) : 0.0;
        mask[q] = e ? 1 : 0;
        fix[q] = e || face ? 1 : 0;
        phi[q] = e ? f : outer;
        const unsigned long long b = e ? abs_bits(f) : 0ull;
        m = b > m ? b : m;
    }
    block_max(m, &sc->rmax);
}

// mqlv::coarse_fix
__global__ void __launch_bounds__(kT) k_coarse_fix(const uint8_t* __restrict__ ffix, int fnx, int fny, int fnz, uint8_t* __restrict__ cfix,
                                                   int cnx, int cny, int cnz) {
    const unsigned t = blockIdx.x * kT + threadIdx.x, n = (unsigned)cnx * (unsigned)cny;
    const int K = block_plane();
    if (t >= n || K >= cnz) return;
    const int I = (int)(t % (unsigned)cnx), J = (int)(t / (unsigned)cnx);
    bool fx = I == 0 || J == 0 || K == 0 || I == cnx - 1 || J == cny - 1 || K == cnz - 1;
    if (!fx) {
        const int i = 2 * I, j = 2 * J, k = 2 * K;
        fx = i >= fnx || j >= fny || k >= fnz || ffix[(size_t)i + (size_t)fnx * ((size_t)j + (size_t)fny * k)] != 0;
    }
    cfix[(size_t)t + (size_t)n * K] = fx ? 1 : 0;
}

// E = -grad phi by central differences (channel.rs:172), one-sided at the faces; w = mask (RF basis) or 0.
// The divisors are h and 2 h alone, so the quotients are formed without a division.
__global__ void __launch_bounds__(kT) k_efield(const double* __restrict__ phi, int nx, int ny, int nz, double h, double inv_h,
                                               const uint8_t* __restrict__ mask, float4* __restrict__ e4) {
    const unsigned t = blockIdx.x * kT + threadIdx.x, n = (unsigned)nx * (unsigned)ny;
    const int k = block_plane();
    if (t >= n || k >= nz) return;
    const int i = (int)(t % (unsigned)nx), j = (int)(t / (unsigned)nx);
    const size_t q = (size_t)t + (size_t)n * k;
    auto diff = [&](int x, int nn, size_t st) {
        const int m = x > 0 ? 1 : 0, p = x + 1 < nn ? 1 : 0;
        const double d = -(phi[q + (p ? st : 0)] - phi[q - (m ? st : 0)]);
        return (float)(m + p == 2 ? mqp::div_rn(d, 2.0 * h, 0.5 * inv_h) : mqp::div_rn(d, h, inv_h));
    };
    const float ex = diff(i, nx, 1), ey = diff(j, ny, (size_t)nx), ez = diff(k, nz, (size_t)n);
    e4[q] = make_float4(ex, ey, ez, mask ? (float)mask[q] : 0.0f);
}

unsigned blocks(size_t n) { return (unsigned)((n + kT - 1) / kT); }
dim3 plane_blocks(size_t per_plane, int planes) {
    const unsigned z = ((unsigned)planes + 65534u) / 65535u;
    return dim3(blocks(per_plane), ((unsigned)planes + z - 1u) / z, z);
}

// one device allocation, handed out in pieces
struct Arena {
    char* base = nullptr;
    size_t size = 0, used = 0;
    cudaStream_t st = nullptr;
    ~Arena() {
        if (st) { cudaStreamSynchronize(st); cudaStreamDestroy(st); }
        if (base) cudaFree(base);
    }
    static size_t up(size_t b) { return (b + 255) & ~(size_t)255; }
    mq_status open(size_t bytes) {
        if (cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking) != cudaSuccess) { cudaGetLastError(); return MQ_ERR_CUDA; }
        if (cudaMalloc(&base, bytes) != cudaSuccess) { cudaGetLastError(); base = nullptr; return MQ_ERR_NOMEM; }
        size = bytes;
        return MQ_OK;
    }
    template <class T>
    T* take(size_t n) {
        T* p = reinterpret_cast<T*>(base + used);
        used += up(n * sizeof(T));
        return p;
    }
};

// device arrays of one solve
struct Problem {
    int nx, ny, nz;
    std::vector<mqlv::Dims> dims;
    std::vector<DLevel> L;
    double *phi, *r, *p, *qv, *rowsum, *plane;
    Scal* sc;
    uint32_t* cnts;
    size_t n() const { return (size_t)nx * ny * nz; }
    bool lists;   // the levels have lists of their free nodes
    static bool can_list(const std::vector<mqlv::Dims>& dims) { return mqlv::count(dims[0]) < ((size_t)1 << 32); }
    static size_t half(const mqlv::Dims& d) { return (size_t)((d.nx - 1) / 2) * (d.ny - 2) * (d.nz - 2); }   // nodes of a colour, at most
    static size_t bytes(const std::vector<mqlv::Dims>& dims, bool lists) {
        size_t b = 0;
        for (size_t l = 0; l < dims.size(); ++l) {
            const size_t m = mqlv::count(dims[l]);
            b += Arena::up(m) + (l ? 3 : 2) * Arena::up(8 * m);   // the finest level's right-hand side is the residual
            if (lists) b += 2 * Arena::up(4 * half(dims[l]));
        }
        b += Arena::up(8 * dims.size());
        const mqlv::Dims& f = dims[0];
        b += 4 * Arena::up(8 * mqlv::count(f)) + Arena::up(8 * (size_t)f.ny * f.nz) + Arena::up(8 * (size_t)f.nz) + Arena::up(sizeof(Scal));
        return b;
    }
    void carve(Arena& A, const std::vector<mqlv::Dims>& d, bool with_lists) {
        dims = d;
        lists = with_lists;
        nx = d[0].nx; ny = d[0].ny; nz = d[0].nz;
        phi = A.take<double>(n()); r = A.take<double>(n()); p = A.take<double>(n()); qv = A.take<double>(n());
        rowsum = A.take<double>((size_t)ny * nz); plane = A.take<double>((size_t)nz); sc = A.take<Scal>(1);
        L.resize(d.size());
        for (size_t l = 0; l < d.size(); ++l) {
            DLevel& v = L[l];
            v.nx = d[l].nx; v.ny = d[l].ny; v.nz = d[l].nz;
            v.fix = A.take<uint8_t>(v.n());
            v.u = A.take<double>(v.n());
            v.r = A.take<double>(v.n());
            v.rhs = l ? A.take<double>(v.n()) : r;
            for (int c = 0; c < 2; ++c) { v.list[c] = lists ? A.take<uint32_t>(half(d[l])) : nullptr; v.cnt[c] = 0; }
        }
        cnts = A.take<uint32_t>(2 * d.size());
    }
};

int grid_blocks(int device) {
    int sms = 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) { cudaGetLastError(); sms = 1; }
    return sms * 8;
}

// Solve P (fix, phi and sc->rmax = max |fixed| of the finest level set on st); *stats but for the time
mq_status solve(Problem& P, double outer_bc, double tol, int device, cudaStream_t st, mq_solve_stats* stats) {
    const int nx = P.nx, ny = P.ny, nz = P.nz, wide = grid_blocks(device);
    const size_t n = P.n(), rows = (size_t)ny * nz;
    Scal h;
    auto read = [&]() -> bool {
        if (cudaMemcpyAsync(&h, P.sc, sizeof(h), cudaMemcpyDeviceToHost, st) != cudaSuccess) return false;
        return cudaStreamSynchronize(st) == cudaSuccess;
    };
    auto as_double = [](unsigned long long b) {
        double v;
        std::memcpy(&v, &b, 8);
        return v;
    };
    for (size_t l = 1; l < P.L.size(); ++l) {
        const DLevel &f = P.L[l - 1], &c = P.L[l];
        k_coarse_fix<<<plane_blocks((size_t)c.nx * c.ny, c.nz), kT, 0, st>>>(f.fix, f.nx, f.ny, f.nz, c.fix, c.nx, c.ny, c.nz);
    }
    // the levels from `low` on run in one block
    size_t low = P.L.size(), nodes = 0;
    while (low > 0 && P.L.size() - low < (size_t)kBottomLevels && nodes + P.L[low - 1].n() <= (size_t)kBottomNodes) nodes += P.L[--low].n();
    // lists for the levels that have kernels of their own, and for the first below, whose right-hand side these form
    std::vector<uint32_t> cnts(2 * P.L.size(), 0u);
    if (P.lists && low > 0) {
        if (cudaMemsetAsync(P.cnts, 0, cnts.size() * sizeof(uint32_t), st) != cudaSuccess) return MQ_ERR_CUDA;
        for (size_t l = 0; l < P.L.size() && l <= low; ++l)
            for (int c = 0; c < 2; ++c) {
                const DLevel& v = P.L[l];
                k_list<<<plane_blocks((size_t)((v.nx - 1) / 2) * (v.ny - 2), v.nz - 2), kT, 0, st>>>(v.fix, v.nx, v.ny, v.nz, c, v.list[c],
                                                                                                  Problem::half(P.dims[l]), P.cnts + 2 * l + c);
            }
        if (cudaMemcpyAsync(cnts.data(), P.cnts, cnts.size() * sizeof(uint32_t), cudaMemcpyDeviceToHost, st) != cudaSuccess) return MQ_ERR_CUDA;
    }
    if (!read()) return MQ_ERR_CUDA;
    for (size_t l = 0; l < P.L.size(); ++l)
        for (int c = 0; c < 2; ++c) P.L[l].cnt[c] = cnts[2 * l + c];
    double scale = std::fmax(as_double(h.rmax), std::fabs(outer_bc));
    if (!(scale > 0)) scale = 1.0;
    const double target = tol * scale;

    Bottom B{};
    for (size_t l = low; l < P.L.size(); ++l) {
        const int x = B.levels++;
        B.nx[x] = P.L[l].nx; B.ny[x] = P.L[l].ny; B.nz[x] = P.L[l].nz; B.fix[x] = P.L[l].fix;
    }
    const int bottom_bytes = (int)(25 * nodes + 8);
    if (cudaFuncSetAttribute(k_bottom, cudaFuncAttributeMaxDynamicSharedMemorySize, 25 * kBottomNodes + 8) != cudaSuccess) return MQ_ERR_CUDA;
    for (size_t l = 0; l < low; ++l)
        if (cudaMemsetAsync(P.L[l].r, 0, P.L[l].n() * sizeof(double), st) != cudaSuccess ||
            cudaMemsetAsync(P.L[l].u, 0, P.L[l].n() * sizeof(double), st) != cudaSuccess)
            return MQ_ERR_CUDA;

    // (a level without a free node of a colour still launches one block)
    auto half = [](const DLevel& lv, int c) {
        return lv.list[c] ? dim3(blocks(lv.cnt[c] ? lv.cnt[c] : 1)) : plane_blocks((size_t)((lv.nx - 1) / 2) * (lv.ny - 2), lv.nz - 2);
    };
    auto gs = [&](DLevel& lv, int col) {
        k_gs<false><<<half(lv, col), kT, 0, st>>>(lv.u, lv.rhs, lv.fix, nullptr, lv.nx, lv.ny, lv.nz, col, lv.list[col], lv.cnt[col]);
    };
    // symmetric V-cycle from u = 0 (Solver::vcycle of the host solver): L0.u = M^-1 r
    std::function<void(size_t)> vcycle = [&](size_t l) {
        DLevel& lv = P.L[l];
        if (l == low) {
            k_bottom<<<1, 1024, bottom_bytes, st>>>(B, lv.rhs, lv.u, 60);
            return;
        }
        if (l + 1 == P.L.size()) {
            k_coarse<<<1, 1024, 0, st>>>(lv.u, lv.rhs, lv.fix, lv.nx, lv.ny, lv.nz, 60);
            return;
        }
        k_gs_first<<<half(lv, 0), kT, 0, st>>>(lv.u, lv.rhs, lv.fix, lv.nx, lv.ny, lv.nz, lv.list[0], lv.cnt[0]);
        gs(lv, 1);
        gs(lv, 0);
        k_gs<true><<<half(lv, 1), kT, 0, st>>>(lv.u, lv.rhs, lv.fix, lv.r, lv.nx, lv.ny, lv.nz, 1, lv.list[1], lv.cnt[1]);
        k_residual<<<half(lv, 0), kT, 0, st>>>(lv.u, lv.rhs, lv.fix, lv.r, lv.nx, lv.ny, lv.nz, lv.list[0], lv.cnt[0]);
        DLevel& c = P.L[l + 1];
        const uint32_t cn = c.cnt[0] + c.cnt[1];
        k_restrict<<<c.list[0] ? dim3(blocks(cn ? cn : 1)) : plane_blocks((size_t)c.nx * c.ny, c.nz), kT, 0, st>>>(
            lv.r, lv.nx, lv.ny, c.rhs, c.fix, c.nx, c.ny, c.nz, c.list[0], c.cnt[0], c.list[1], c.cnt[1]);
        vcycle(l + 1);
        k_prolong<<<half(lv, 0), kT, 0, st>>>(c.u, c.nx, c.ny, lv.u, lv.fix, lv.nx, lv.ny, lv.nz, lv.list[0], lv.cnt[0]);
        for (int s = 0; s < 2; ++s) { gs(lv, 1); gs(lv, 0); }
    };
    auto true_residual = [&]() -> bool {
        cudaMemsetAsync(P.sc, 0, sizeof(Scal), st);
        k_true_residual<<<wide, kT, 0, st>>>(P.phi, P.L[0].fix, P.r, nx, ny, n, P.sc);
        return read();
    };
    const unsigned rb = (unsigned)((rows + kRows - 1) / kRows);
    auto dot_r_u = [&](Sum what) {
        k_rows<false><<<rb, kT + 32, 0, st>>>(P.r, P.L[0].u, nullptr, nullptr, nx, ny, rows, P.rowsum);
        k_planes<<<nz, 32, 0, st>>>(P.rowsum, ny, P.plane, P.sc, what);
    };

    if (!true_residual()) return MQ_ERR_CUDA;
    double rmax = as_double(h.rmax);
    int it = 0;
    const int max_it = 2000;
    bool converged = rmax <= target;
    while (!converged && it < max_it) {
        vcycle(0);
        cudaMemcpyAsync(P.p, P.L[0].u, n * sizeof(double), cudaMemcpyDeviceToDevice, st);
        dot_r_u(RZ0);
        int inner = 0;
        while (it < max_it) {
            k_rows<true><<<rb, kT + 32, 0, st>>>(P.p, nullptr, P.L[0].fix, P.qv, nx, ny, rows, P.rowsum);
            k_planes<<<nz, 32, 0, st>>>(P.rowsum, ny, P.plane, P.sc, ALPHA);
            k_cg_update<<<wide, kT, 0, st>>>(P.phi, P.r, P.p, P.qv, P.L[0].fix, n, it == 0, P.sc);
            if (!read()) return MQ_ERR_CUDA;
            if (!(h.pq > 0)) break;
            rmax = as_double(h.rmax);
            ++it;
            ++inner;
            if (rmax <= target || inner >= 200) break;
            vcycle(0);
            dot_r_u(BETA);
            k_cg_dir<<<blocks(n), kT, 0, st>>>(P.p, P.L[0].u, n, P.sc);
        }
        if (!true_residual()) return MQ_ERR_CUDA;
        rmax = as_double(h.rmax);
        converged = rmax <= target;
        if (!converged && inner == 0) break;
    }
    if (cudaGetLastError() != cudaSuccess) return MQ_ERR_CUDA;
    if (stats) {
        stats->iterations = it;
        stats->converged = converged ? 1 : 0;
        stats->final_residual = rmax / scale;
    }
    return converged ? MQ_OK : MQ_ERR_NOT_CONVERGED;
}

bool have_device(int device) {
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || device < 0 || device >= ndev) { cudaGetLastError(); return false; }
    return true;
}

// Gives a host array its pages (their content stays) while the GPU works: the copy into a fresh array
// would wait for each. Where the kernel cannot, or no thread is to be had, the copy does it as before.
struct Pages {
    std::thread t;
    void give(void* a, size_t na, void* b, size_t nb) try {
        t = std::thread([=] { one(a, na); one(b, nb); });
    } catch (...) {
    }
    static void one(void* p, size_t n) {
        const uintptr_t pg = (uintptr_t)sysconf(_SC_PAGESIZE), lo = ((uintptr_t)p + pg - 1) / pg * pg, hi = ((uintptr_t)p + n) / pg * pg;
#ifdef MADV_POPULATE_WRITE
        if (p && hi > lo) madvise(reinterpret_cast<void*>(lo), hi - lo, MADV_POPULATE_WRITE);
#endif
    }
    void wait() { if (t.joinable()) t.join(); }
    ~Pages() { wait(); }
};

}  // namespace

extern "C" {

mq_status mq_laplace_solve_device(int32_t nx, int32_t ny, int32_t nz, const uint8_t* mask, const double* fixed,
                                  double outer_bc, double tol, int32_t device, double* phi, mq_solve_stats* stats) {
    return mq_laplace_solve_device_lists(nx, ny, nz, mask, fixed, outer_bc, tol, device, 1, phi, stats);
}

mq_status mq_laplace_solve_device_lists(int32_t nx, int32_t ny, int32_t nz, const uint8_t* mask, const double* fixed, double outer_bc,
                                        double tol, int32_t device, int32_t lists, double* phi, mq_solve_stats* stats) {
    if (nx < 3 || ny < 3 || nz < 3 || !mask || !fixed || !phi || !(tol > 0)) return MQ_ERR_INVALID;
    if (!have_device(device)) return MQ_ERR_NO_DEVICE;
    if (cudaSetDevice(device) != cudaSuccess) return MQ_ERR_CUDA;
    const auto t0 = std::chrono::steady_clock::now();
    const std::vector<mqlv::Dims> dims = mqlv::hierarchy(nx, ny, nz);
    const size_t n = mqlv::count(dims[0]);
    Arena A;
    Problem P;
    const bool listed = lists && Problem::can_list(dims);
    mq_status s = A.open(Problem::bytes(dims, listed) + Arena::up(n));
    if (s != MQ_OK) return s;
    P.carve(A, dims, listed);
    uint8_t* dmask = A.take<uint8_t>(n);
    if (cudaMemcpyAsync(dmask, mask, n, cudaMemcpyHostToDevice, A.st) != cudaSuccess) return MQ_ERR_CUDA;
    if (cudaMemcpyAsync(P.p, fixed, n * sizeof(double), cudaMemcpyHostToDevice, A.st) != cudaSuccess) return MQ_ERR_CUDA;
    if (cudaMemsetAsync(P.sc, 0, sizeof(Scal), A.st) != cudaSuccess) return MQ_ERR_CUDA;
    k_problem<<<grid_blocks(device), kT, 0, A.st>>>(dmask, P.p, outer_bc, nx, ny, nz, P.L[0].fix, P.phi, P.sc);
    s = solve(P, outer_bc, tol, device, A.st, stats);
    if (s != MQ_OK && s != MQ_ERR_NOT_CONVERGED) return s;
    if (cudaMemcpyAsync(phi, P.phi, n * sizeof(double), cudaMemcpyDeviceToHost, A.st) != cudaSuccess) return MQ_ERR_CUDA;
    if (cudaStreamSynchronize(A.st) != cudaSuccess) return MQ_ERR_CUDA;
    if (stats) stats->seconds = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
    return s;
}

}  // extern "C"

// a basis of a channel geometry (mq_channel_basis_ex on a device): electrodes, solve and E field on the GPU
mq_status mq_channel_basis_device(const mq_geom* g, int32_t basis, double tol, int32_t device, float* e4, double* phi_out,
                                  mq_solve_stats* stats) {
    int32_t d[3];
    if (mq_geom_dims(g, d) != MQ_OK || !e4 || basis < 0 || basis > 5 || !(tol > 0) || d[0] < 3 || d[1] < 3) return MQ_ERR_INVALID;
    if (!have_device(device)) return MQ_ERR_NO_DEVICE;
    if (cudaSetDevice(device) != cudaSuccess) return MQ_ERR_CUDA;
    const auto t0 = std::chrono::steady_clock::now();
    const std::vector<mqlv::Dims> dims = mqlv::hierarchy(d[0], d[1], d[2]);
    const size_t n = mqlv::count(dims[0]);
    const double outer = basis == MQ_BASIS_DC_BOX ? 1.0 : 0.0;
    Arena A;
    Problem P;
    const bool listed = Problem::can_list(dims);
    mq_status s = A.open(Problem::bytes(dims, listed) + Arena::up(n));
    if (s != MQ_OK) return s;
    P.carve(A, dims, listed);
    uint8_t* mask = A.take<uint8_t>(n);
    if (cudaMemsetAsync(P.sc, 0, sizeof(Scal), A.st) != cudaSuccess) return MQ_ERR_CUDA;
    k_channel<<<grid_blocks(device), kT, 0, A.st>>>(*g, mqgeo::layers_of(g), basis, outer, d[0], d[1], d[2], mask, P.L[0].fix, P.phi, P.sc);
    Pages pages;
    if (n >= (1u << 18)) pages.give(e4, n * 16, phi_out, n * 8);
    s = solve(P, outer, tol, device, A.st, stats);
    pages.wait();
    if (s != MQ_OK) {
        // the potential reached so far, as the host path leaves it
        if (s == MQ_ERR_NOT_CONVERGED && phi_out &&
            (cudaMemcpyAsync(phi_out, P.phi, n * sizeof(double), cudaMemcpyDeviceToHost, A.st) != cudaSuccess ||
             cudaStreamSynchronize(A.st) != cudaSuccess))
            return MQ_ERR_CUDA;
        if (stats) stats->seconds = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
        return s;
    }
    // the field takes the place of p and q, which lie side by side
    static_assert(sizeof(float4) == 2 * sizeof(double), "field node");
    float4* e = reinterpret_cast<float4*>(P.p);
    const double h = g->h_mm * 1e-3;
    k_efield<<<plane_blocks((size_t)d[0] * d[1], d[2]), kT, 0, A.st>>>(P.phi, d[0], d[1], d[2], h, 1.0 / h,
                                                                      basis == MQ_BASIS_RF ? mask : nullptr, e);
    if (cudaGetLastError() != cudaSuccess) return MQ_ERR_CUDA;
    if (stats) {   // as before: the solve, without the field
        cudaStreamSynchronize(A.st);
        stats->seconds = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
    }
    if (phi_out && cudaMemcpyAsync(phi_out, P.phi, n * sizeof(double), cudaMemcpyDeviceToHost, A.st) != cudaSuccess) return MQ_ERR_CUDA;
    if (cudaMemcpyAsync(e4, e, n * sizeof(float4), cudaMemcpyDeviceToHost, A.st) != cudaSuccess) return MQ_ERR_CUDA;
    return cudaStreamSynchronize(A.st) == cudaSuccess ? MQ_OK : MQ_ERR_CUDA;
}

MQ_CHECK_READER(mq_check_read_solve)
