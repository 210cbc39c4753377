// Batched mixed-precision ion-trajectory engine for sm_103a.
//
// Same physics as the FP64 integrator (simulation/mqviz/src/world.rs:498-536 with chsim's
// switches, simulation/chsim/src/channel.metal:70-124), re-shaped for throughput:
//   * persistent workers: each lane pulls ions from a device work queue (one warp-
//     aggregated atomic per refill) and advances its ion until it finishes or has done
//     `chunk` steps; survivors are appended to the next launch's list by warp-ballot
//     compaction, so every launch starts with dense warps (chsim tc_filter + tc_tail,
//     channel_tiled.metal:341-482);
//   * positions in grid units and velocities in cells per step, each an FP32 double-float
//     (compensated two-sum accumulator); field nodes, interpolation and collision
//     kinematics in FP32;
//   * a second kernel with four lanes per ion for the lists that leave the chip idle: short ones, and
//     the last ions of a long one;
//   * fields as interleaved node records of 96 bytes (256-bit loads) or 48 bytes, by grid size;
//     the 8 corners of the ion's cell x {RF, DC, AC} held in registers and reloaded only when
//     the ion changes cell (the cached conductor bits of the corners give the nearest-node
//     crash test), with an optional L1 prefetch of the cell the ion is heading for;
//   * RF / AC phase as exact 64-bit fixed-point turn accumulators (phase = offset +
//     step * f * dt mod 1), evaluated with an FP32 quarter-turn polynomial;
//   * Philox-4x32-10 counter RNG keyed by the ion's 64-bit key, counter = step (thermal candidates
//     and collisions) or 4-step window (legacy collisions: two blocks per window); thermal
//     candidates drawn against the majorant |v| + E|V| (mqx::thermal_partner), which samples the
//     reference's collision process with 2 to 3.4 times fewer candidates than its |v| + 6 s_gas;
//   * device injection with the FP64 injection's draws and FP32 transforms (k_inject_mixed).
#include "mq_mixed.h"
#include "mq_check.h"
#include "mq_mixmath.h"

#include <cstring>
#include <vector>

namespace mqmix {
namespace {

using mqd::DevGrid;
using mqd::DevIons;
using namespace mqx;

constexpr unsigned FULL = 0xffffffffu;

constexpr int kMaxLegs = 10;         // lane-group launches of one round

struct Ctrs {                       // device counters
    uint32_t head;                  // work-queue head of the current launch
    uint32_t count[2];              // live-list lengths (ping-pong)
    uint32_t open;                  // ions the current launch has not finished
    uint32_t head_g[kMaxLegs];      // queue heads of the lane-group launches, beyond their first ions
    uint32_t handed[kMaxLegs + 2];  // ions handed to each of them, by k_mixed or by the one before
    unsigned long long steps;       // executed ion-steps
    unsigned long long cell_loads;  // cell-cache fills (a cell's 8 corners each)
    unsigned long long queued;      // ions queued over the call's launches
};

// ---------------------------------------------------------------- FP32 turn-based sine
// sin / cos Taylor polynomials on [-pi/4, pi/4] (coefficients (-1)^k/(2k+1)!, (-1)^k/(2k)!)
__device__ __forceinline__ float sinp(float x) {
    float z = x * x;
    float p = fmaf(z, 0x1.71de3ap-19f, -0x1.a01a02p-13f);
    p = fmaf(z, p, 0x1.111112p-7f);
    p = fmaf(z, p, -0x1.555556p-3f);
    return fmaf(x * z, p, x);
}
__device__ __forceinline__ float cosp(float x) {
    float z = x * x;
    float p = fmaf(z, -0x1.27e4fcp-22f, 0x1.a01a02p-16f);
    p = fmaf(z, p, -0x1.6c16c2p-10f);
    p = fmaf(z, p, 0x1.555556p-5f);
    return fmaf(z * z, p, fmaf(z, -0.5f, 1.0f));
}
// sin and cos of 2 pi P / 2^64 for a 64-bit fixed-point phase in turns
__device__ __forceinline__ void turn_sincos(uint64_t P, float& so, float& co) {
    int64_t r = (int64_t)(P << 2);                      // remainder of 4*phase in [-1/2, 1/2) quarter turns
    uint32_t q = (uint32_t)(P >> 62) + (r < 0 ? 1u : 0u);
    float x = (float)(int32_t)(r >> 32) * 0x1.921fb6p-32f;   // (pi/2) * 2^-32
    float s = sinp(x), c = cosp(x);
    float vs = (q & 1u) ? c : s, vc = (q & 1u) ? -s : c;
    so = (q & 2u) ? -vs : vs;
    co = (q & 2u) ? -vc : vc;
}
// one step of the drive: rotate (s, c) by the per-step angle (cw, sw)
__device__ __forceinline__ void rotate(float& s, float& c, float cw, float sw) {
    const float s2 = fmaf(s, cw, c * sw);
    c = fmaf(c, cw, -(s * sw));
    s = s2;
}

// ---------------------------------------------------------------- cell cache
// Node records, interleaved by field component d (RF, combined DC, AC of one component side by side, so
// that a lane which needs one component reads one piece), each with the conductor bits of the cell
// based at the node:
//   narrow  48 B: float4 [3q + d] = {RF, DC, AC, bits}: a cell is 4 runs of 2 records (x neighbours);
//   wide    96 B: float4 [6q + 2d] = {RF, RF', DC, DC'}, [6q + 2d + 1] = {AC, AC', bits, 0}, the primes from
//           the node above (z + 1): a cell is 2 runs of 2 records, 12 sectors and 12 256-bit loads (4 for
//           a lane of a group), and the values come in the pairs that two-at-a-time arithmetic takes.
// Wide records are faster where the cell reloads hit L2, slower on fine grids whose gathers reach HBM
// and pay for twice the footprint.
// Narrow: a corner lies in the slot of its node's parity, not of its place in the cell, so a move to the next
// cell along an axis replaces the far face's four slots and leaves the near face where it is; the order of
// an axis's two slots goes into the interpolation. These grids' fills are bound by L1 (24 reads of 16 bytes for
// each lane, every other step), and 92 in 100 moves are along one axis: 0.050 mm study of a million ions 40.6 ms
// with whole fills, which want neighbours' lines in L1 and so one block per SM, 39.1 with half fills, 30.5
// with two blocks of 255 registers (three of 168 spill: 33.9). Wide records come from L2 past L1, and there
// the slots' extra instructions cost more than half the reads give (sweep 55.8 -> 60.8 ms).
struct Cell {
    float R[3][8], D[3][8], A[3][8];   // corner values per field and component, corner or slot q = a + 2b + 4c
    uint32_t bits[8];                   // narrow: conductor bits of the cell based at each slot's node
    int32_t ci, cj, ck;
    float fci, fcj, fck;                // the same cell as floats (no int -> float conversion per step)
    uint32_t mask;                      // conductor bit per corner
};

// node indices are 32-bit (the host refuses grids with 3 x nodes >= 2^32): less address arithmetic in
// the divergent reload path (measured about 1% on the sweep)
__device__ __forceinline__ uint32_t node_of(const MixBatch& B, int32_t ci, int32_t cj, int32_t ck) {
    return (uint32_t)ci + (uint32_t)B.nx * ((uint32_t)cj + (uint32_t)B.ny * (uint32_t)ck);
}

// the same without allocating the lines in L1 (they are fetched from L2 into registers)
__device__ __forceinline__ void ld256_na(const float4* p, float4& a, float4& b) {
    asm("ld.global.nc.L1::no_allocate.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
        : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w), "=f"(b.x), "=f"(b.y), "=f"(b.z), "=f"(b.w) : "l"(p));
}

// 16 bytes of a narrow record, where p is set
__device__ __forceinline__ void ld_narrow(const float4* n, bool p, float& r, float& d, float& a, uint32_t& bits) {
    asm("{.reg .pred p; setp.ne.u32 p, %4, 0; @p ld.global.nc.v4.b32 {%0,%1,%2,%3}, [%5];}"
        : "+f"(r), "+f"(d), "+f"(a), "+r"(bits) : "r"((uint32_t)p), "l"(n));
}

// NEAREST (the reference's legacy field mode: the field of the cell's lowest corner, t = 0) reads
// only that corner's record, which also holds the cell's conductor bits: one record per fill.
// A narrow fill reads the slots that hold another node than the new cell's, and leaves the conductor bits to
// cell_mask (so that nothing waits for the reads here).
template <bool WIDE, bool NEAREST>
__device__ __forceinline__ void load_cell(const float4* __restrict__ nodes, const MixBatch& B, int32_t ci, int32_t cj,
                                          int32_t ck, Cell& c) {
    const uint32_t sy = (uint32_t)B.nx, sz = (uint32_t)B.nx * (uint32_t)B.ny;
    uint32_t base = node_of(B, ci, cj, ck);
    uint32_t m = 0;
    if (WIDE) {
        base = (uint32_t)MQ_CHK_SPAN(base, NEAREST ? 1u : sy + 2u, (size_t)sz * (size_t)B.nz, MQ_SITE_MIX_CELL);
        const float4* const p0 = nodes + (size_t)6 * base;
        const float4* const p2 = p0 + (size_t)6 * sy;
#pragma unroll
        for (int q = 0; q < (NEAREST ? 1 : 4); ++q) {
            const float4* p = ((q & 2) ? p2 : p0) + 6 * (q & 1);
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                float4 u, v;
                // left out of L1: these grids' fills hit L2, and the kernel's other data keeps the L1
                // (5% on the sweep)
                if (NEAREST) ld256(p + 2 * d, u, v);
                else ld256_na(p + 2 * d, u, v);
                c.R[d][q] = u.x; c.D[d][q] = u.z; c.A[d][q] = v.x;
                if (!NEAREST) { c.R[d][q + 4] = u.y; c.D[d][q + 4] = u.w; c.A[d][q + 4] = v.y; }
                if (q == 0 && d == 0) m = __float_as_uint(v.z);   // conductor bits of the cell's corners
            }
        }
    } else if (NEAREST) {
        const uint32_t o = (uint32_t)MQ_CHK_SPAN(3u * base, 3u, 3u * (size_t)sz * (size_t)B.nz, MQ_SITE_MIX_CELL);
        const float4 x = __ldg(nodes + o), y = __ldg(nodes + o + 1), z = __ldg(nodes + o + 2);
        c.R[0][0] = x.x; c.R[1][0] = y.x; c.R[2][0] = z.x;
        c.D[0][0] = x.y; c.D[1][0] = y.y; c.D[2][0] = z.y;
        c.A[0][0] = x.z; c.A[1][0] = y.z; c.A[2][0] = z.z;
        m = __float_as_uint(x.w);
    } else {
        // nodes of each parity along the axes, and whether the slots hold others
        const int32_t i0 = ci + (ci & 1), i1 = ci | 1, j0 = cj + (cj & 1), j1 = cj | 1, k0 = ck + (ck & 1), k1 = ck | 1;
        const bool sx0 = i0 != c.ci + (c.ci & 1), sx1 = i1 != (c.ci | 1), sy0 = j0 != c.cj + (c.cj & 1), sy1 = j1 != (c.cj | 1);
        const bool sz0 = k0 != c.ck + (c.ck & 1), sz1 = k1 != (c.ck | 1);
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const bool p = ((q & 1) ? sx1 : sx0) || ((q & 2) ? sy1 : sy0) || ((q & 4) ? sz1 : sz0);
            uint32_t o = 3u * node_of(B, (q & 1) ? i1 : i0, (q & 2) ? j1 : j0, (q & 4) ? k1 : k0);
            o = (uint32_t)MQ_CHK_SPAN(o, 3u, 3u * (size_t)sz * (size_t)B.nz, MQ_SITE_MIX_CELL);
            ld_narrow(nodes + o, p, c.R[0][q], c.D[0][q], c.A[0][q], c.bits[q]);
            uint32_t pad;
            ld_narrow(nodes + o + 1, p, c.R[1][q], c.D[1][q], c.A[1][q], pad);
            ld_narrow(nodes + o + 2, p, c.R[2][q], c.D[2][q], c.A[2][q], pad);
        }
    }
    c.ci = ci; c.cj = cj; c.ck = ck; c.mask = m;
    c.fci = (float)ci; c.fcj = (float)cj; c.fck = (float)ck;
}

__device__ __forceinline__ uint32_t cell_mask(const Cell& c) {
    const bool px = c.ci & 1, py = c.cj & 1, pz = c.ck & 1;
    const uint32_t m0 = py ? (px ? c.bits[3] : c.bits[2]) : (px ? c.bits[1] : c.bits[0]);
    const uint32_t m1 = py ? (px ? c.bits[7] : c.bits[6]) : (px ? c.bits[5] : c.bits[4]);
    return pz ? m1 : m0;
}

// pull the 4 corner runs of a cell into L1 ahead of use
template <bool WIDE>
__device__ __forceinline__ void prefetch_cell(const float4* nodes, const MixBatch& B, int32_t ci, int32_t cj, int32_t ck) {
    const uint32_t sy = (uint32_t)B.nx, sz = (uint32_t)B.nx * (uint32_t)B.ny;
    const uint32_t base = node_of(B, ci, cj, ck);
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        if (WIDE) {   // two runs of two 96-byte records
            const float4* p = nodes + (size_t)6 * (base + ((r & 2) ? sy : 0u) + (uint32_t)(r & 1));
            asm volatile("prefetch.global.L1 [%0];" ::"l"(p));
            asm volatile("prefetch.global.L1 [%0];" ::"l"(p + 5));
        } else {
            const float4* p = nodes + 3 * (base + ((r & 1) ? sy : 0) + ((r & 2) ? sz : 0));
            asm volatile("prefetch.global.L1 [%0];" ::"l"(p));
            asm volatile("prefetch.global.L1 [%0];" ::"l"(p + 5));
        }
    }
}

// lo + t (hi - lo) of an axis's two values. SLOTS: odd says that the second is the lower node's, and t is
// negative then; hi - lo is the same number but for its sign, so that only a zero's sign can differ.
template <bool SLOTS>
__device__ __forceinline__ float lerp2(float t, bool odd, float f0, float f1) { return fmaf(t, f1 - f0, SLOTS && odd ? f1 : f0); }

// E = a_rf RF(t) + DC(t) + a_ac AC(t): corner values combined first, then one trilinear pass
template <bool SLOTS>
__device__ __forceinline__ float field_comp(const float R[8], const float D[8], const float A[8], float a_rf, float a_ac,
                                            float tx, float ty, float tz, bool ox, bool oy, bool oz) {
    float F[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) F[q] = fmaf(a_rf, R[q], fmaf(a_ac, A[q], D[q]));
    const float c00 = lerp2<SLOTS>(tx, ox, F[0], F[1]), c10 = lerp2<SLOTS>(tx, ox, F[2], F[3]);
    const float c01 = lerp2<SLOTS>(tx, ox, F[4], F[5]), c11 = lerp2<SLOTS>(tx, ox, F[6], F[7]);
    const float c0 = lerp2<SLOTS>(ty, oy, c00, c10), c1 = lerp2<SLOTS>(ty, oy, c01, c11);
    return lerp2<SLOTS>(tz, oz, c0, c1);
}

// (xh + xl) - (th + tl) for a double-float position and threshold, as the sign-exact difference of
// two double-floats: xh - th is exact wherever the two are within a factor of 2 of each other (which
// covers every position close enough to the threshold for the low parts to matter), so the sign of
// the result is the sign of the unrounded difference there
__device__ __forceinline__ float df_diff(float xh, float xl, float th, float tl) {
    return __fadd_rn(__fsub_rn(xh, th), __fsub_rn(xl, tl));
}

// an ion's counters to its state, its position and velocity to the working state
__device__ __forceinline__ void put_ion(const DevIons& io, float* __restrict__ keep, uint32_t n_all, uint32_t id, uint32_t n, uint32_t ncoll,
                                        int32_t leg, int32_t status, const float xh[3], const float xl[3], const float uh[3],
                                        const float ul[3]) {
    io.steps[id] = n; io.ncoll[id] = ncoll; io.leg[id] = leg; io.status[id] = status;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        keep[(size_t)(0 + d) * n_all + id] = xh[d]; keep[(size_t)(3 + d) * n_all + id] = xl[d];
        keep[(size_t)(6 + d) * n_all + id] = uh[d]; keep[(size_t)(9 + d) * n_all + id] = ul[d];
    }
}

// ---------------------------------------------------------------- the persistent worker
// What bounds it: with 96-byte records the latency of a step's chain and of the cell fills (on nearly every step of a
// warp some lane needs one) at 12 or 16 warps per SM; with 48-byte records on larger grids the L1 reads of the
// fills. So registers are kept for the cell, and all that only every fourth step, a collision or the end of a
// flight reads lies in shared memory. BLOCKS: blocks per SM that the registers are cut for: 3 with wide records, 4
// for long lists, 2 with narrow ones, which then need no spills, or 3 with legacy collisions (resident_blocks() has the rules).
// Measured, wide with registers only / tables in shared memory at 3 / at 4 blocks: sweep of 4.2 million ions 51.1 / 51.9 /
// 48.7 ms, 40,000 legacy ions 15.4 / 15.0 / 15.0; narrow, 0.050 mm study 30.5 / 27.6 at 2 blocks (34.4 at 3).
template <bool LEGACY, bool PREFETCH, bool WIDE, bool NEAREST, int BLOCKS>
__global__ void __launch_bounds__(128, BLOCKS)
k_mixed(const float4* __restrict__ nodes, MixBatch B, const MixJob* __restrict__ jobs, DevIons io,
        const uint32_t* __restrict__ list_in, uint32_t* __restrict__ list_out, Ctrs* ctr, int in_slot, uint32_t chunk,
        float* __restrict__ keep, const uint64_t* __restrict__ kph, uint32_t n_all, uint2* __restrict__ hand, uint32_t hand_at) {
    // keep: the working state of every ion of the call in grid units, double-float position and
    // velocity (12 floats per ion, structure of arrays over n_all), filled from the FP64 states by
    // k_init_list and written back to them by k_unstage, so this kernel does no FP64 arithmetic;
    // kph: the RF / AC phase offsets as 64-bit fixed-point turns (two arrays of n_all)
    // The job constants only the collision branches read are staged per lane in shared memory at
    // refill, so those divergent branches do not wait on a global load (1.5% on the sweep, 5% on the
    // legacy-collision scan, against re-reading the job record there).
    __shared__ float sj_sgas[128], sj_mr[128], sj_floor[128], sj_mfp[128];
    // What a window of four steps needs besides the positions, made at its first step for all of them: the drive
    // amplitudes, and the candidates' uniforms or the legacy collisions' words; and what only that and the ends of
    // a flight read.
    __shared__ float2 s_amp[4][128];
    __shared__ float s_uni[LEGACY ? 1 : 4][128];
    __shared__ uint2 s_word[LEGACY ? 4 : 1][128];
    __shared__ uint64_t s_ph[3][128];       // phases at the next window's start, AC turns per step
    __shared__ float4 s_drv[128];           // AC amplitude, rotation
    __shared__ uint2 s_key[128];
    __shared__ uint32_t s_id[128], s_n0[128], s_nc[128];
    __shared__ unsigned long long s_tot[128];
    const uint32_t tid = threadIdx.x;
    s_tot[tid] = 0;
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t count = ctr->count[in_slot];
    if (count <= hand_at) return;   // the lane-group launch takes them
    uint32_t* count_out = &ctr->count[in_slot ^ 1];

    // lanes that take ions: all 32 when the list fills the grid, else the warp's even share of it
    const uint32_t warps = gridDim.x * (blockDim.x >> 5);
    bool have = false, drained = lane >= (count + warps - 1) / warps;
    uint32_t n = 0, stop = 0;           // the ion's step count, and the one to put it away at
    int32_t leg = 0;
    float xh[3], xl[3], uh[3], ul[3];
    const uint64_t Wrf = ((uint64_t)B.w_rf_hi << 32) | B.w_rf_lo;
    float kick = 0.f, cand_aa = 0.f, cand_b = 0.f;
    // The drive is evaluated exactly from the fixed-point phases at every step that is a multiple of 4 and rotated
    // in between, so rounding cannot build up, and one Philox block (legacy: two) serves four steps.
    float2 amp = make_float2(0.f, 0.f);   // drive amplitudes of the next step
    auto window = [&]() {
        const uint64_t prf = s_ph[0][tid], pac = s_ph[1][tid], wac = s_ph[2][tid];
        const float4 dv = s_drv[tid];
        float s, c, sa, ca;
        turn_sincos(prf, s, c);
        turn_sincos(pac, sa, ca);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            s_amp[q][tid] = make_float2(B.v_rf * s, dv.x * sa);
            if (q < 3) { rotate(s, c, B.cw_rf, B.sw_rf); rotate(sa, ca, dv.y, dv.z); }
        }
        s_ph[0][tid] = prf + 4u * Wrf;
        s_ph[1][tid] = pac + 4u * wac;
        const uint2 key = s_key[tid];
        if (!LEGACY) {
            const uint4 r = philox(key.x, key.y, n >> 2, 0u, 0u, 0u);
            s_uni[0][tid] = unif(r.x); s_uni[LEGACY ? 0 : 1][tid] = unif(r.y);
            s_uni[LEGACY ? 0 : 2][tid] = unif(r.z); s_uni[LEGACY ? 0 : 3][tid] = unif(r.w);
        } else {
            const uint4 ra = philox(key.x, key.y, n >> 2, 2u, 0u, 0u), rb = philox(key.x, key.y, n >> 2, 3u, 0u, 0u);
            s_word[0][tid] = make_uint2(ra.x, ra.y); s_word[LEGACY ? 1 : 0][tid] = make_uint2(ra.z, ra.w);
            s_word[LEGACY ? 2 : 0][tid] = make_uint2(rb.x, rb.y); s_word[LEGACY ? 3 : 0][tid] = make_uint2(rb.z, rb.w);
        }
    };
    uint32_t iter = 0;
    uint32_t loads = 0;                 // cell-cache fills of this lane
    Cell c;
#pragma unroll
    for (int d = 0; d < 3; ++d) { xh[d] = xl[d] = uh[d] = ul[d] = 0.f; }
    c.ci = c.cj = c.ck = -1; c.mask = 0;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        c.bits[q] = 0;
#pragma unroll
        for (int d = 0; d < 3; ++d) c.R[d][q] = c.D[d][q] = c.A[d][q] = 0.f;
    }
    c.fci = c.fcj = c.fck = __int_as_float(0x7fc00000);   // NaN: differs from every floored position

    // Queue traffic is warp-synchronous and happens once every 4 iterations: survivors that ended in
    // the last 4 iterations are appended to the next launch's list, then lanes without an ion are
    // refilled (a lane that finished waits at most 3 iterations; 1.8% on the sweep and 3% on the
    // legacy scan against ballots every iteration).
    bool append = false, ended = false;
    for (;;) {
      if ((iter & 3u) == 0u) {
        // ---- ions that ended; when the queue is empty and few are left, they go on in lane groups
        const unsigned em = __ballot_sync(FULL, ended);
        if (em && lane == 0) atomicSub(&ctr->open, (uint32_t)__popc(em));
        ended = false;
        if ((iter & 31u) == 0u && (__any_sync(FULL, drained) || (iter & 255u) == 0u)) {
            // (lanes beyond the warp's share are drained from the start, and blocks may come after others have
            // ended, so that the queue is empty is read off its head; the queue's last ions may fill warps whose lanes
            // never come to it again, so every warp looks once in a while: 60,000 ions with legacy collisions, 58,368
            // at once, 3,000 steps 10.4 -> 7.8 ms)
            const uint32_t open = __shfl_sync(FULL, *(volatile uint32_t*)&ctr->open, 0);
            const uint32_t head = __shfl_sync(FULL, *(volatile uint32_t*)&ctr->head, 0);
            if (open <= hand_at && head >= count) {
                if (have) {
                    const uint32_t id = s_id[tid], done = n - s_n0[tid];
                    hand[MQ_CHK(atomicAdd(&ctr->handed[0], 1u), hand_at, MQ_SITE_MIX_HAND)] = make_uint2(id, done);
                    put_ion(io, keep, n_all, id, n, s_nc[tid], leg, 0, xh, xl, uh, ul);
                    s_tot[tid] += done;
                    have = false;
                }
                drained = true;
            }
        }
        // ---- warp-ballot compaction of survivors into the next launch's list
        const unsigned am = __ballot_sync(FULL, append);
        if (am) {
            const int leader = __ffs(am) - 1;
            uint32_t base = 0;
            if ((int)lane == leader) base = atomicAdd(count_out, (uint32_t)__popc(am));
            base = __shfl_sync(FULL, base, leader);
            if (append) list_out[MQ_CHK(base + __popc(am & ((1u << lane) - 1u)), n_all, MQ_SITE_MIX_LIST_OUT)] = s_id[tid];
        }
        append = false;
        // ---- refill: one warp-aggregated atomic hands out queue slots to lanes without an ion
        const unsigned need = __ballot_sync(FULL, !have && !drained);
        if (need) {
            const int leader = __ffs(need) - 1;
            uint32_t base = 0;
            if ((int)lane == leader) base = atomicAdd(&ctr->head, (uint32_t)__popc(need));
            base = __shfl_sync(FULL, base, leader);
            if (!have && !drained) {
                const uint32_t slot = base + __popc(need & ((1u << lane) - 1u));
                if (slot < count) {
                    const uint32_t id = (uint32_t)MQ_CHK(__ldg(list_in + slot), n_all, MQ_SITE_MIX_ION);
                    const MixJob J = jobs[io.jid[id]];
                    sj_sgas[tid] = J.s_gas;
                    sj_mr[tid] = J.mr;
                    sj_floor[tid] = J.floor_v;
                    sj_mfp[tid] = J.mfp_mean;
                    kick = J.kick; cand_aa = J.cand_a * J.cand_a; cand_b = J.cand_b;
                    n = io.steps[id]; leg = io.leg[id];
                    s_id[tid] = id; s_n0[tid] = n; s_nc[tid] = io.ncoll[id];
                    s_drv[tid] = make_float4(J.use_ac ? J.v_ac : 0.0f, J.cw_ac, J.sw_ac, 0.0f);
#pragma unroll
                    for (int d = 0; d < 3; ++d) {
                        xh[d] = keep[(size_t)(0 + d) * n_all + id]; xl[d] = keep[(size_t)(3 + d) * n_all + id];
                        uh[d] = keep[(size_t)(6 + d) * n_all + id]; ul[d] = keep[(size_t)(9 + d) * n_all + id];
                    }
                    // phase = offset + step * w (mod 1) in 64-bit fixed point, at the start of the ion's window
                    const uint64_t wac = ((uint64_t)J.w_ac_hi << 32) | J.w_ac_lo;
                    s_ph[0][tid] = kph[id] + (uint64_t)(n & ~3u) * Wrf;
                    s_ph[1][tid] = kph[(size_t)n_all + id] + (uint64_t)(n & ~3u) * wac;
                    s_ph[2][tid] = wac;
                    const uint64_t key = io.rng[id];
                    s_key[tid] = make_uint2((uint32_t)key, (uint32_t)(key >> 32));
                    // An ion at a multiple of 4 steps (every fresh ion) first steps on an iteration that makes its window
                    if (n & 3u) {
                        window();
                        if (WIDE) amp = s_amp[n & 3u][tid];
                    }
                    c.ck = -4;   // nothing held is of use
                    load_cell<WIDE, NEAREST>(nodes, B, clampi(__float2int_rd(xh[0]), 0, B.nx - 2), clampi(__float2int_rd(xh[1]), 0, B.ny - 2),
                              clampi(__float2int_rd(xh[2]), 0, B.nz - 2), c);
                    ++loads;
                    stop = n >= B.max_steps ? n + 1u : B.max_steps - n < chunk ? B.max_steps : n + chunk;
                    have = true;
                } else {
                    drained = true;
                }
            }
        }
        if (!__any_sync(FULL, have)) break;
      }

        // A lane steps its ion only when the ion's step count is congruent to the warp's
        // iteration counter mod 4 (a freshly loaded ion waits at most 3 iterations).  Every
        // warp-uniform event below (Philox refresh and exact drive re-sync, each 4 iterations)
        // then falls on the same steps of every ion, whatever the scheduling, so per-ion
        // results are reproducible bit for bit.
        const bool act = have && (((iter ^ n) & 3u) == 0u);
        if ((iter & 3u) == 0u && act) {
            window();
            if (WIDE) amp = s_amp[0][tid];
        }
        const uint32_t now = iter & 3u;
        ++iter;
        if (act) {
            // ---- field at the current position
            float tx = 0.f, ty = 0.f, tz = 0.f;
            if (!NEAREST) {
                tx = __fadd_rn(__fsub_rn(xh[0], c.fci), xl[0]);
                ty = __fadd_rn(__fsub_rn(xh[1], c.fcj), xl[1]);
                tz = __fadd_rn(__fsub_rn(xh[2], c.fck), xl[2]);
            }
            if (!WIDE) amp = s_amp[now][tid];
            const float a_rf = amp.x, a_ac = amp.y;
            if (WIDE) amp = s_amp[(now + 1u) & 3u][tid];   // the next step's (at the window's end made anew)
            float E[3];
            const bool ox = c.ci & 1, oy = c.cj & 1, oz = c.ck & 1;
            if (!NEAREST && !WIDE) {
                tx = ox ? -tx : tx;
                ty = oy ? -ty : ty;
                tz = oz ? -tz : tz;
            }
#pragma unroll
            for (int d = 0; d < 3; ++d)
                E[d] = NEAREST ? fmaf(a_rf, c.R[d][0], fmaf(a_ac, c.A[d][0], c.D[d][0]))   // = field_comp at t = 0
                               : field_comp<!WIDE>(c.R[d], c.D[d], c.A[d], a_rf, a_ac, tx, ty, tz, ox, oy, oz);
            // ---- kick (compensated) and drift (compensated)
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                float inc = __fadd_rn(__fmul_rn(kick, E[d]), ul[d]);
                two_sum(uh[d], inc, uh[d], ul[d]);
                float s, e;
                fast_two_sum(xh[d], uh[d], s, e);
                e = __fadd_rn(e, __fadd_rn(xl[d], ul[d]));
                fast_two_sum(s, e, xh[d], xl[d]);
            }
            // ---- cell of the new position: its records are asked for before the collisions, which move no ion,
            //      so that their way from L2 is covered by these (55.8 -> 53.0 ms on the sweep); and an L1 prefetch of
            //      the cell one more step ahead. Cell changes are found on floored floats; an ion outside the box
            //      (the unclamped cell index leaving [0, n-2]) has ended and needs no cell
            const float ffi = floorf(xh[0]), ffj = floorf(xh[1]), ffk = floorf(xh[2]);
            bool out = false;
            if (ffi != c.fci || ffj != c.fcj || ffk != c.fck) {
                out = ffi < 0.0f || ffj < 0.0f || ffk < 0.0f || ffi > B.lim_x - 1.0f || ffj > B.lim_y - 1.0f || ffk > B.lim_z - 1.0f;
                if (!out) {
                    load_cell<WIDE, NEAREST>(nodes, B, __float2int_rz(ffi), __float2int_rz(ffj), __float2int_rz(ffk), c);
                    c.fci = ffi; c.fcj = ffj; c.fck = ffk;
                    ++loads;
                }
            }
            if (PREFETCH && !NEAREST) {
                const int32_t pi = clampi(__float2int_rd(xh[0] + uh[0]), 0, B.nx - 2);
                const int32_t pj = clampi(__float2int_rd(xh[1] + uh[1]), 0, B.ny - 2);
                const int32_t pk = clampi(__float2int_rd(xh[2] + uh[2]), 0, B.nz - 2);
                if (pi != c.ci || pj != c.cj || pk != c.ck) prefetch_cell<WIDE>(nodes, B, pi, pj, pk);
            }
            if (!WIDE && !NEAREST) c.mask = cell_mask(c);
            const uint32_t nprev = n;
            n += 1;
            // ---- collisions
            if (!LEGACY) {
                const float u0 = s_uni[LEGACY ? 0 : now][tid];
                // candidate if u0 < cand_a |u| + cand_b = n sigma dt (|v| + E|V|), tested on squares
                // (no square root per step); see thermal_partner for why E|V| bounds the rate
                const float um2 = fmaf(uh[0], uh[0], fmaf(uh[1], uh[1], uh[2] * uh[2]));
                const float du = u0 - cand_b;
                if (du < 0.0f || du * du < cand_aa * um2) {
                    const float um = sqrtf(um2);
                    const float s_gas = sj_sgas[tid], mr = sj_mr[tid];
                    // two Philox blocks per candidate, drawn side by side: the first for the gas
                    // partner and the acceptance, the second for the scattering direction
                    const uint2 key = s_key[tid];
                    const uint4 r0 = philox(key.x, key.y, nprev, 1u, 0u, 0u);
                    const uint4 r1 = philox(key.x, key.y, nprev, 2u, 0u, 0u);
                    const float u2v = B.u2v_f;
                    float v[3] = {uh[0] * u2v, uh[1] * u2v, uh[2] * u2v};
                    float gv[3], vm_sum;
                    thermal_partner(r0, s_gas, um * u2v, v, gv, vm_sum);
                    const float gl = sqrtf(fmaf(gv[0], gv[0], fmaf(gv[1], gv[1], gv[2] * gv[2])));
                    if (unif16(r0.w & 0xffffu) * vm_sum < gl) {
                        const float cth = 2.0f * unif(r1.x) - 1.0f;
                        float sp, cp;
                        angle_sincos(unif(r1.y), &sp, &cp);
                        const float sn = sqrtf(fmaxf(0.0f, 1.0f - cth * cth));
                        const float nn[3] = {sn * cp, sn * sp, cth};
                        const float v2u = B.v2u_f;
#pragma unroll
                        for (int d = 0; d < 3; ++d) {
                            float vn = fmaf(mr * gl, nn[d], fmaf(-mr, gv[d], v[d]));
                            uh[d] = vn * v2u; ul[d] = 0.0f;
                        }
                        s_nc[tid] += 1u;
                    }
                }
            } else {
                // a collision is due every ~4 steps per ion, so some lane of the warp needs one on
                // almost every iteration: every lane computes it and keeps it only where it is due,
                // with selects instead of a divergent branch
                leg -= 1;
                const bool due = leg <= 0;
                {
                    const float mr = sj_mr[tid], floor_v = sj_floor[tid], mfp_mean = sj_mfp[tid];
                    // two 32-bit words of this window step: cos(theta) from the top 24 bits of the
                    // first, the free path from the top 24 of the second, phi from their low bytes
                    const uint2 word = s_word[LEGACY ? now : 0][tid];
                    const uint32_t wa = word.x, wb = word.y;
                    const float u2v = B.u2v_f;
                    float v[3] = {uh[0] * u2v, uh[1] * u2v, uh[2] * u2v};
                    const float vm = sqrtf(fmaf(v[0], v[0], fmaf(v[1], v[1], v[2] * v[2])));
                    const bool hit = due && vm > floor_v;
                    const float cth = 2.0f * unif(wa) - 1.0f;
                    float sp, cp;
                    angle_sincos(unif16(((wa & 0xffu) << 8) | (wb & 0xffu)), &sp, &cp);
                    const float sn = sqrtf(fmaxf(0.0f, 1.0f - cth * cth));
                    const float dd[3] = {sn * cp, sn * sp, cth};
                    const float v2u = B.v2u_f;
#pragma unroll
                    for (int d = 0; d < 3; ++d) {
                        const float vn = fmaf(mr * vm, dd[d], v[d] * (1.0f - mr));
                        v[d] = hit ? vn : v[d];
                        uh[d] = hit ? vn * v2u : uh[d];
                        ul[d] = hit ? 0.0f : ul[d];
                    }
                    if (hit) s_nc[tid] += 1u;
                    const float mfp = -__logf(fmaxf(unif(wb), 1e-7f)) * mfp_mean;
                    const float vn = sqrtf(fmaf(v[0], v[0], fmaf(v[1], v[1], v[2] * v[2])));
                    // free path in steps with the hardware's approximate division (within 2 ulp; the
                    // floored count moves by one step in rare ties, a few ions in 10^5; 3.8% on the
                    // legacy scan against two IEEE divisions)
                    const float st = floorf(__fdividef(mfp, fmaxf(vn, 1e-3f) * B.dt_f));
                    const int32_t nl = st < 1.0f ? 1 : (st < 2147483520.0f ? (int32_t)st : 2147483647);
                    leg = due ? nl : leg;
                }
            }
            // ---- termination tests: exit, return, box, conductor, timeout
            // (the loss-surface planes - exit, return and the crash window - are crossed on the full
            // double-float position against the double-float thresholds; the box test is the
            // unclamped cell index leaving [0, n-2])
            // A plane farther away than the low parts reach cannot be crossed, so the exact test runs
            // only close to it; the crash window matters only in a cell with
            // a conductor corner (most cells have none).
            int32_t status = 0;
            if (xh[2] > B.z_exit_near && df_diff(xh[2], xl[2], B.z_exit_h, B.z_exit_l) > 0.0f) status = 3;
            else if (xh[2] < B.z_ret_near && df_diff(xh[2], xl[2], B.z_ret_h, B.z_ret_l) < 0.0f) status = 2;
            else if (out) status = 4;
            else {
                if (c.mask != 0u && df_diff(xh[2], xl[2], B.cz0_h, B.cz0_l) > 0.0f &&
                    df_diff(xh[2], xl[2], B.cz1_h, B.cz1_l) < 0.0f) {
                    const float fx = __fadd_rn(__fsub_rn(xh[0], c.fci), xl[0]);
                    const float fy = __fadd_rn(__fsub_rn(xh[1], c.fcj), xl[1]);
                    const float fz = __fadd_rn(__fsub_rn(xh[2], c.fck), xl[2]);
                    const uint32_t q = (fx >= 0.5f ? 1u : 0u) | (fy >= 0.5f ? 2u : 0u) | (fz >= 0.5f ? 4u : 0u);
                    if ((c.mask >> q) & 1u) status = 1;
                }
            }
            if (status != 0 || n >= stop) {
                if (status == 0 && n >= B.max_steps) status = 5;
                // ---- write back: counters to the ion states, position and velocity to the working
                //      state (k_unstage turns it into the FP64 state when the caller wants that)
                put_ion(io, keep, n_all, s_id[tid], n, s_nc[tid], leg, status, xh, xl, uh, ul);
                ended = true;
                s_tot[tid] += n - s_n0[tid];
                append = status == 0;
                have = false;
            }
        }
    }
    unsigned long long steps_total = s_tot[tid];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        steps_total += __shfl_down_sync(FULL, steps_total, o);
        loads += __shfl_down_sync(FULL, loads, o);
    }
    if (lane == 0 && steps_total) atomicAdd(&ctr->steps, steps_total);
    if (lane == 0 && loads) atomicAdd(&ctr->cell_loads, (unsigned long long)loads);
}

// ---------------------------------------------------------------- lane groups
// The same steps with four lanes per ion, for lists that leave the chip idle (few ions, or the last
// ones of a large batch): there the time of a step is what counts, not lanes. Lanes 0..2 each hold
// one axis (position, velocity, cell, and that component of the cell's field records: one read per
// corner pair); lane 3 repeats lane 0. The fractions and velocities that all axes need go round by
// shuffles. What depends on the step count alone is prepared 16 steps at a time, a part in each lane,
// and lies in shared memory: the drive amplitudes, and the candidates' uniforms or the legacy
// collisions' directions and free paths. Every operation is k_mixed's, on the same numbers, so an
// ion's states do not depend on which kernel steps it.
// What bounds it: the latency of one step's chain (position -> fractions -> field -> kick -> position)
// and, with many ions to a warp, the reload of some ion's cell on nearly every step; so the chain is kept
// short (one vote clears most steps) and registers few. A step takes 0.27 us for up to 608 ions,
// 0.44 for 4,864 and 0.57 for 19,456 (S14 grid), where the one-lane kernel takes 0.8 to 1.1; from there
// on the one-lane kernel's 58,368 ions in flight win (0.86 us a step for 26,000), so longer lists start with it.
// Measured when these groups came, whole run_batch calls, without -> with them: 1,000 ions at one point
// 2.25 -> 1.04 ms; mass scan of 25,000 short-lived ions 1.26 -> 0.82; Fig. 4 legacy scan 21.2 -> 10.8;
// S14 sweep of 62,000 ions 76.7 -> 39.9; sweep of 4.2 million ions 63.7 -> 55.6.
// One block per SM, as many warps as the registers hold (16 at 128 a thread; 24 at 80 where the nearest
// node's record is the whole cell).
constexpr int group_block(bool nearest) { return nearest ? 768 : 512; }
// Warps per SM that share the ions: two a scheduler, which hide each other's waits; more only once these
// would hold over eight ions each (9,728 ions of the S14 grid: 0.49 us a step with 8 warps, 0.51 with 16)
constexpr uint32_t kGroupFirst = 8;

// Shared floats of a group: 16 steps x {RF, AC} amplitudes, then 16 x {uniform} or 16 x {direction, free path}
// (and 4 more, so that the 8 groups of a warp read different banks)
__host__ __device__ constexpr int group_floats(bool legacy) { return 36 + (legacy ? 64 : 16); }
// two FP32 operations in one instruction, each rounded as alone
__device__ __forceinline__ uint64_t pack2(float a, float b) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void unpack2(uint64_t v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ uint64_t sub2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

template <bool LEGACY, bool WIDE, bool NEAREST>
__global__ void __launch_bounds__(group_block(NEAREST), 1)
k_mixed_group(const float4* __restrict__ nodes, MixBatch B, const MixJob* __restrict__ jobs, DevIons io,
              const uint32_t* __restrict__ list_in, uint2* __restrict__ hand, uint32_t* __restrict__ list_out, Ctrs* ctr,
              int in_slot, uint32_t chunk, int leg_no, uint32_t leg_steps, float* __restrict__ keep,
              const uint64_t* __restrict__ kph, uint32_t n_all, uint32_t hand_at) {
    constexpr int NQ = NEAREST ? 1 : 4;
    const uint32_t lane = threadIdx.x & 31u, gl = lane & 3u, base = lane & ~3u, warp = threadIdx.x >> 5;
    // Legs of one round: each steps its ions by at most leg_steps and hands on those that are neither ended
    // nor at the round's `chunk` steps; the next starts with full warps again. The first leg takes a short
    // list whole, of a long one what k_mixed handed on.
    const bool direct = leg_no == 0 && ctr->count[in_slot] <= hand_at;
    const uint32_t count = direct ? ctr->count[in_slot] : ctr->handed[leg_no];
    if (count == 0) return;
    const uint2* const from = hand + (size_t)(leg_no & 1) * hand_at;
    uint2* const to = hand + (size_t)((leg_no & 1) ^ 1) * hand_at;
    const uint32_t groups = gridDim.x * (blockDim.x >> 2);
    const uint32_t warps = blockDim.x >> 5, full = (count + 8u * gridDim.x - 1u) / (8u * gridDim.x);
    const uint32_t lead = full < kGroupFirst ? kGroupFirst : full > warps ? warps : full;
    const uint32_t first = warp < lead ? ((lane >> 2) * lead + warp) * gridDim.x + blockIdx.x
                                       : (8u * lead + (lane >> 2) * (warps - lead) + warp - lead) * gridDim.x + blockIdx.x;
    extern __shared__ __align__(16) float group_sm[];
    float* const drive = group_sm + (size_t)(threadIdx.x >> 2) * group_floats(LEGACY);
    float* const draws = drive + 32;
    const int d = gl == 3u ? 0 : (int)gl;
    const bool is_z = gl == 2u, is_ac = (gl & 1u) != 0u;
    const int32_t top = (d == 0 ? B.nx : d == 1 ? B.ny : B.nz) - 2;
    const float lim = d == 0 ? B.lim_x : d == 1 ? B.lim_y : B.lim_z;
    const uint32_t sy = (uint32_t)B.nx, sz = (uint32_t)B.nx * (uint32_t)B.ny;
    const uint32_t stride = gl == 0u ? 1u : gl == 1u ? sy : gl == 2u ? sz : 0u;
    const size_t row = (size_t)(WIDE ? 6u : 3u) * sy, layer = (size_t)3 * sz;   // to the y and z neighbours' records
    // positions that no plane or face can end: beyond them the exact tests run
    const float in_lo = is_z ? fmaxf(B.z_ret_near, 0.0f) : 0.0f, in_hi = is_z ? fminf(B.z_exit_near, lim - 0.0625f) : lim - 0.0625f;

    // Every lane of the warp runs every step together (the shuffles then need no lane masks): a group
    // without an ion moves a particle of speed 1 that no force acts on, and keeps nothing. (Zeros,
    // infinities and NaN would take the slow branch of the square roots, every step, for the whole warp.)
    bool have = false, waits = false, drained = false, fresh = true;
    bool idle = true;                    // some group of the warp has no ion under way
    uint32_t id = 0, jid = 0, n = 0, n0 = 0, done = 0, stop = 0, ncoll = 0, k0 = 0, k1 = 0, mask = 0, loads = 0;
    int32_t leg = 0;
    float xh = 0.f, xl = 0.f, uh = 1.f, ul = 0.f, fc = 0.f;
    // the component's RF, DC and AC values: corner q in the low half, q + 4 (z + 1) in the high one
    uint64_t R[NQ], D[NQ], A[NQ];
    uint64_t P = 0, W = 0;
    float cw = 1.f, sw = 0.f, amp = 0.f, kick = 0.f, ca2 = 0.f, cand_b = 0.f;
    float mr = 0.f, floor_v = 0.f, mfp_mean = 0.f;     // legacy collisions
    unsigned long long steps_total = 0;
#pragma unroll
    for (int q = 0; q < NQ; ++q) R[q] = D[q] = A[q] = 0;

    // node records of the cell that holds the group's position, the lane's component
    auto fill = [&](bool go) {
        const int32_t ci = clampi(__float2int_rd(xh), 0, top);
        uint32_t o = (uint32_t)ci * stride;
        o += __shfl_xor_sync(FULL, o, 1);
        o += __shfl_xor_sync(FULL, o, 2);
        if (!go) return;
        fc = (float)ci;
        ++loads;
        // the cell's highest record read: with narrow records one layer up, which wide ones hold
        o = (uint32_t)MQ_CHK_SPAN(o, NEAREST ? 1u : (WIDE ? 0u : sz) + sy + 2u, (size_t)sz * (size_t)B.nz, MQ_SITE_MIX_CELL);
        const float4* const p = nodes + (size_t)(WIDE ? 6u : 3u) * o + (WIDE ? 2 : 1) * d;
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
            const float4* pq = p + ((q & 1) ? (WIDE ? 6 : 3) : 0) + ((q & 2) ? row : 0);
            float4 u, v;
            if (WIDE) {
                ld256(pq, u, v);
                if (q == 0) mask = __float_as_uint(v.z);
            } else {
                const float4 r = __ldg(pq), t = NEAREST ? make_float4(0.f, 0.f, 0.f, 0.f) : __ldg(pq + layer);
                u = make_float4(r.x, t.x, r.y, t.y);
                v = make_float4(r.z, t.z, 0.f, 0.f);
                if (q == 0) mask = __float_as_uint(r.w);
            }
            R[q] = pack2(u.x, u.y); D[q] = pack2(u.z, u.w); A[q] = pack2(v.x, v.y);
        }
    };
    // tables of the 16-step block that holds step n (P is the drive phase at its start): each lane one
    // window of four steps of the draws, and two windows of its drive (lanes 0, 1 the first two, 2, 3 the others):
    // exact at a window's start, then rotated
    auto block = [&]() {
        const uint32_t w = ((n >> 4) << 2) + gl;
        if (LEGACY) {
            // a collision at window step q takes words 2q and 2q + 1 of the window's two blocks: cos(theta)
            // from the top 24 bits of the first, the free path from the top 24 of the second, phi from their low bytes
            const uint4 ra = philox(k0, k1, w, 2u, 0u, 0u), rb = philox(k0, k1, w, 3u, 0u, 0u);
            const uint32_t wa[4] = {ra.x, ra.z, rb.x, rb.z}, wb[4] = {ra.y, ra.w, rb.y, rb.w};
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const float cth = 2.0f * unif(wa[q]) - 1.0f;
                float sp, cp;
                angle_sincos(unif16(((wa[q] & 0xffu) << 8) | (wb[q] & 0xffu)), &sp, &cp);
                const float sn = sqrtf(fmaxf(0.0f, 1.0f - cth * cth));
                reinterpret_cast<float4*>(draws)[4u * gl + q] =
                    make_float4(sn * cp, sn * sp, cth, -__logf(fmaxf(unif(wb[q]), 1e-7f)));
            }
        } else {
            const uint4 r = philox(k0, k1, w, 0u, 0u, 0u);
            reinterpret_cast<float4*>(draws)[gl] = make_float4(unif(r.x), unif(r.y), unif(r.z), unif(r.w));
        }
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const uint32_t q0 = ((gl & 2u) + (uint32_t)k) * 4u;
            float s, c;
            turn_sincos(P + (uint64_t)q0 * W, s, c);
#pragma unroll
            for (uint32_t q = 0; q < 4u; ++q) {
                drive[2u * (q0 + q) + (gl & 1u)] = amp * s;
                rotate(s, c, cw, sw);
            }
        }
        P += 16u * W;
    };

    // exact termination tests: exit, return, box, conductor, time-out
    auto test = [&](float ff) {
        int32_t status = 0;
        uint32_t zf = 0;
        if (is_z) {
            if (xh > B.z_exit_near && df_diff(xh, xl, B.z_exit_h, B.z_exit_l) > 0.0f) zf = 3;
            else if (xh < B.z_ret_near && df_diff(xh, xl, B.z_ret_h, B.z_ret_l) < 0.0f) zf = 2;
            if (df_diff(xh, xl, B.cz0_h, B.cz0_l) > 0.0f && df_diff(xh, xl, B.cz1_h, B.cz1_l) < 0.0f) zf |= 4;
        }
        zf = __shfl_sync(FULL, zf, base + 2);
        const unsigned out = (__ballot_sync(FULL, ff < 0.0f || ff > lim - 1.0f) >> base) & 7u;
        const unsigned corner = (__ballot_sync(FULL, __fadd_rn(__fsub_rn(xh, fc), xl) >= 0.5f) >> base) & 7u;
        if (zf & 3u) status = (int32_t)(zf & 3u);
        else if (out) status = 4;
        else if (mask != 0u && (zf & 4u) && ((mask >> corner) & 1u)) status = 1;
        else if (n >= B.max_steps) status = 5;
        if (have && (!LEGACY || n != n0) && (status != 0 || n >= stop)) {
            if (gl < 3u) {
                keep[(size_t)d * n_all + id] = xh; keep[(size_t)(3 + d) * n_all + id] = xl;
                keep[(size_t)(6 + d) * n_all + id] = uh; keep[(size_t)(9 + d) * n_all + id] = ul;
            }
            if (gl == 0u) {
                io.steps[id] = n; io.ncoll[id] = ncoll; io.leg[id] = leg; io.status[id] = status;
                done += n - n0;
                if (status == 0 && done < chunk)
                    to[MQ_CHK(atomicAdd(&ctr->handed[leg_no + 1], 1u), hand_at, MQ_SITE_MIX_HAND)] = make_uint2(id, done);
                else if (status == 0)
                    list_out[MQ_CHK(atomicAdd(&ctr->count[in_slot ^ 1], 1u), n_all, MQ_SITE_MIX_LIST_OUT)] = id;
                steps_total += n - n0;
            }
            have = false;
            kick = 0.f; uh = 1.f; xh = xl = ul = 0.f;
        }
        idle = __any_sync(FULL, !have);
    };

    // Drive amplitudes of the step. Legacy steps read the next one's ahead (Fig. 4 scan 10.71 -> 10.56 ms: the read is
    // at the head of the step's chain); thermal ones do not (S14 sweep 39.0 against 39.4 ms with it).
    float2 a2 = make_float2(0.f, 0.f);
    for (uint32_t iter = 0;; ++iter) {
        if (idle) {
            // ---- groups without an ion take the next one of the list
            const unsigned need = __ballot_sync(FULL, !have && !waits && !drained && gl == 0u);
            if (need && (iter & 15u) == 0u) {
                uint32_t slot = first;
                const unsigned later = __ballot_sync(FULL, !have && !waits && !drained && gl == 0u && !fresh);
                if (later) {
                    uint32_t q = 0;
                    const int leader = __ffs(later) - 1;
                    if ((int)lane == leader) q = atomicAdd(&ctr->head_g[leg_no], (uint32_t)__popc(later));
                    q = __shfl_sync(FULL, q, leader) + groups;
                    if (!fresh) slot = q + __popc(later & ((1u << base) - 1u));
                }
                if (!have && !waits && !drained) {
                    fresh = false;
                    if (slot >= count) drained = true;
                    else {
                        done = 0;
                        if (direct) id = list_in[slot];
                        else { const uint2 e = from[slot]; id = e.x; done = e.y; }
                        id = (uint32_t)MQ_CHK(id, n_all, MQ_SITE_MIX_ION);
                        n = io.steps[id];
                        waits = true;
                    }
                }
            }
            // An ion starts when its step count is congruent to the warp's counter mod 16, so that every
            // block of words and phases begins on the same iteration for all of the warp's ions
            const bool start = waits && ((iter ^ n) & 15u) == 0u;
            if (__any_sync(FULL, start)) {
                if (start) {
                    have = true;
                    waits = false;
                    jid = io.jid[id];
                    const MixJob& J = jobs[jid];
                    kick = J.kick; ca2 = J.cand_a * J.cand_a; cand_b = J.cand_b;
                    if (LEGACY) { mr = J.mr; floor_v = J.floor_v; mfp_mean = J.mfp_mean; }
                    const uint64_t Wrf = ((uint64_t)B.w_rf_hi << 32) | B.w_rf_lo, Wac = ((uint64_t)J.w_ac_hi << 32) | J.w_ac_lo;
                    W = is_ac ? Wac : Wrf;
                    cw = is_ac ? J.cw_ac : B.cw_rf;
                    sw = is_ac ? J.sw_ac : B.sw_rf;
                    amp = is_ac ? (J.use_ac ? J.v_ac : 0.0f) : B.v_rf;
                    n0 = n; ncoll = io.ncoll[id]; leg = io.leg[id];
                    // the step to stop at: the time-out (one step at least), the end of the round or of the leg
                    uint32_t left = n < B.max_steps ? B.max_steps - n : 1u;
                    left = left < chunk - done ? left : chunk - done;
                    stop = n + (left < leg_steps ? left : leg_steps);
                    xh = keep[(size_t)d * n_all + id]; xl = keep[(size_t)(3 + d) * n_all + id];
                    uh = keep[(size_t)(6 + d) * n_all + id]; ul = keep[(size_t)(9 + d) * n_all + id];
                    P = kph[(is_ac ? (size_t)n_all : 0) + id] + (uint64_t)(n & ~15u) * W;
                    const uint64_t key = io.rng[id];
                    k0 = (uint32_t)key; k1 = (uint32_t)(key >> 32);
                    if (n & 15u) block();
                }
                fill(start);
                __syncwarp();
                if (LEGACY) a2 = reinterpret_cast<const float2*>(drive)[iter & 15u];
            }
            idle = __any_sync(FULL, !have && !drained);
            if (!idle && !__any_sync(FULL, have)) break;
        }
        if ((iter & 15u) == 0u) {
            __syncwarp();
            block();
            __syncwarp();
            if (LEGACY) a2 = reinterpret_cast<const float2*>(drive)[0];
        }
        const uint32_t now = iter & 15u;
        if (!LEGACY) a2 = reinterpret_cast<const float2*>(drive)[now];
        const float a_rf = a2.x, a_ac = a2.y;
        if (LEGACY) a2 = reinterpret_cast<const float2*>(drive)[(now + 1u) & 15u];   // at the block's end made anew
        // ---- field component at the current position: as field_comp, two corners an instruction
        float E;
        if (NEAREST) {
            float r, di, ai, hi;
            unpack2(R[0], r, hi); unpack2(D[0], di, hi); unpack2(A[0], ai, hi);
            E = fmaf(a_rf, r, fmaf(a_ac, ai, di));
        } else {
            const float t = __fadd_rn(__fsub_rn(xh, fc), xl);
            const float tx = __shfl_sync(FULL, t, base), ty = __shfl_sync(FULL, t, base + 1), tz = __shfl_sync(FULL, t, base + 2);
            const uint64_t ar2 = pack2(a_rf, a_rf), aa2 = pack2(a_ac, a_ac);
            uint64_t F[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) F[q] = fma2(ar2, R[q % NQ], fma2(aa2, A[q % NQ], D[q % NQ]));
            const uint64_t tx2 = pack2(tx, tx), ty2 = pack2(ty, ty);
            const uint64_t x0 = fma2(tx2, sub2(F[1], F[0]), F[0]), x1 = fma2(tx2, sub2(F[3], F[2]), F[2]);
            float c0, c1;
            unpack2(fma2(ty2, sub2(x1, x0), x0), c0, c1);
            E = fmaf(tz, c1 - c0, c0);
        }
        // Legacy collisions come every few steps and most warps hold many ions, so nearly every step has a new
        // cell: the tests of a position wait for its records here, where the field needs them anyway
        if (LEGACY && __any_sync(FULL, have && n != n0 && (xh < in_lo || xh > in_hi || mask != 0u || n >= stop))) test(floorf(xh));
        // ---- kick and drift, compensated
        {
            const float inc = __fadd_rn(__fmul_rn(kick, E), ul);
            two_sum(uh, inc, uh, ul);
            float r, e;
            fast_two_sum(xh, uh, r, e);
            e = __fadd_rn(e, __fadd_rn(xl, ul));
            fast_two_sum(r, e, xh, xl);
        }
        n += have ? 1u : 0u;   // a waiting ion's count stays: its start is found by it
        // ---- what the end of the step may have to deal with: a collision, another cell, a limit
        const float ux = __shfl_sync(FULL, uh, base), uy = __shfl_sync(FULL, uh, base + 1), uz = __shfl_sync(FULL, uh, base + 2);
        bool coll;
        float um2 = 0.0f;
        if (!LEGACY) {
            const float u0 = draws[now];
            um2 = fmaf(ux, ux, fmaf(uy, uy, uz * uz));
            const float du = u0 - cand_b;
            coll = have && (du < 0.0f || du * du < ca2 * um2);
        } else {
            leg -= 1;
            coll = have && leg <= 0;
        }
        const float ff = floorf(xh);
        const bool moved = have && ff != fc;
        bool edge = !LEGACY && have && (xh < in_lo || xh > in_hi || mask != 0u || n >= stop);
        if (!LEGACY && !__any_sync(FULL, coll || moved || edge)) continue;
        if (LEGACY) {
            const unsigned ch = __ballot_sync(FULL, moved);
            if (ch) fill(((ch >> base) & 15u) != 0u);
        }
        if (__any_sync(FULL, coll)) {
            if (!LEGACY) {
                // the candidate's two Philox blocks, one in even lanes, one in odd
                const uint4 r = philox(k0, k1, n - 1u, 1u + (gl & 1u), 0u, 0u);
                uint4 r0;
                r0.x = __shfl_sync(FULL, r.x, base); r0.y = __shfl_sync(FULL, r.y, base);
                r0.z = __shfl_sync(FULL, r.z, base); r0.w = __shfl_sync(FULL, r.w, base);
                const uint32_t r1x = __shfl_sync(FULL, r.x, base + 1), r1y = __shfl_sync(FULL, r.y, base + 1);
                if (coll) {
                    const float s_gas = jobs[jid].s_gas, mr_ = jobs[jid].mr;
                    const float um = sqrtf(um2);
                    const float u2v = B.u2v_f;
                    const float v[3] = {ux * u2v, uy * u2v, uz * u2v};
                    float gv[3], vm_sum;
                    thermal_partner(r0, s_gas, um * u2v, v, gv, vm_sum);
                    const float gm = sqrtf(fmaf(gv[0], gv[0], fmaf(gv[1], gv[1], gv[2] * gv[2])));
                    if (unif16(r0.w & 0xffffu) * vm_sum < gm) {
                        const float cth = 2.0f * unif(r1x) - 1.0f;
                        float sp, cp;
                        angle_sincos(unif(r1y), &sp, &cp);
                        const float sn = sqrtf(fmaxf(0.0f, 1.0f - cth * cth));
                        const float nn = d == 0 ? sn * cp : d == 1 ? sn * sp : cth;
                        const float gd = d == 0 ? gv[0] : d == 1 ? gv[1] : gv[2], vd = d == 0 ? v[0] : d == 1 ? v[1] : v[2];
                        const float vn = fmaf(mr_ * gm, nn, fmaf(-mr_, gd, vd));
                        uh = vn * B.v2u_f;
                        ul = 0.0f;
                        ncoll += 1;
                    }
                }
            } else {
                const float4 dr = reinterpret_cast<const float4*>(draws)[now];   // direction, -ln u of the free path
                const float dd[3] = {dr.x, dr.y, dr.z};
                const float u2v = B.u2v_f;
                float v[3] = {ux * u2v, uy * u2v, uz * u2v};
                const float vm = sqrtf(fmaf(v[0], v[0], fmaf(v[1], v[1], v[2] * v[2])));
                const bool hit = coll && vm > floor_v;
                const float v2u = B.v2u_f;
                float own_v = 0.0f;
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    const float vn = fmaf(mr * vm, dd[k], v[k] * (1.0f - mr));
                    v[k] = hit ? vn : v[k];
                    if (k == d) own_v = vn;
                }
                uh = hit ? own_v * v2u : uh;
                ul = hit ? 0.0f : ul;
                ncoll += hit ? 1u : 0u;
                const float mfp = dr.w * mfp_mean;
                const float vn = sqrtf(fmaf(v[0], v[0], fmaf(v[1], v[1], v[2] * v[2])));
                const float st = floorf(__fdividef(mfp, fmaxf(vn, 1e-3f) * B.dt_f));
                const int32_t nl = st < 1.0f ? 1 : (st < 2147483520.0f ? (int32_t)st : 2147483647);
                leg = coll ? nl : leg;
            }
        }
        // ---- cell of the new position
        if (!LEGACY) {
            const unsigned ch = __ballot_sync(FULL, moved);
            if (ch) {
                fill(((ch >> base) & 15u) != 0u);
                edge = edge || (have && mask != 0u);
            }
        }
        // ---- termination tests
        if (!LEGACY && __any_sync(FULL, edge)) test(ff);
    }
    if (gl != 0u) loads = 0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        steps_total += __shfl_down_sync(FULL, steps_total, o);
        loads += __shfl_down_sync(FULL, loads, o);
    }
    if (lane == 0) {
        if (steps_total) atomicAdd(&ctr->steps, steps_total);
        if (loads) atomicAdd(&ctr->cell_loads, (unsigned long long)loads);
    }
}

// interleave RF | combined DC | AC by component into node records of `stride` float4 (once per DC
// configuration and record width); the spare w of each holds the conductor bits of the 8 corners of
// the cell whose lowest corner is this node (bit a + 2b + 4c), so a cell reload reads its crash mask
// in one word
__global__ void k_pack_nodes(const float4* __restrict__ rf, const float4* __restrict__ dc, const float4* __restrict__ ac,
                             float4* __restrict__ nodes, size_t n, int32_t nx, int32_t ny, int32_t nz, int stride) {
    const size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= n) return;
    const float4 r = rf[q], d = dc[q], a = ac[q];
    const size_t sy = (size_t)nx, sz = (size_t)nx * (size_t)ny;
    const int32_t i = (int32_t)(q % sy), j = (int32_t)((q / sy) % (size_t)ny), k = (int32_t)(q / sz);
    uint32_t m = 0;
    if (i < nx - 1 && j < ny - 1 && k < nz - 1)
        for (int c = 0; c < 8; ++c)
            m |= (rf[q + (size_t)(c & 1) + ((c & 2) ? sy : 0) + ((c & 4) ? sz : 0)].w > 0.5f ? 1u : 0u) << c;
    const float w = __uint_as_float(m);
    if (stride == 3) {
        nodes[3 * q] = make_float4(r.x, d.x, a.x, w);
        nodes[3 * q + 1] = make_float4(r.y, d.y, a.y, w);
        nodes[3 * q + 2] = make_float4(r.z, d.z, a.z, w);
    } else {
        const size_t t = k < nz - 1 ? q + sz : q;   // a cell's upper corners; the top layer bases no cell
        const float4 rt = rf[t], dt = dc[t], at = ac[t];
        nodes[6 * q] = make_float4(r.x, rt.x, d.x, dt.x);
        nodes[6 * q + 1] = make_float4(a.x, at.x, w, 0.f);
        nodes[6 * q + 2] = make_float4(r.y, rt.y, d.y, dt.y);
        nodes[6 * q + 3] = make_float4(a.y, at.y, w, 0.f);
        nodes[6 * q + 4] = make_float4(r.z, rt.z, d.z, dt.z);
        nodes[6 * q + 5] = make_float4(a.z, at.z, w, 0.f);
    }
}

// ---------------------------------------------------------------- injection for the mixed engine
// The draws of mqp::inject_one (Ion::inject, world.rs:407-422, with chsim's launches,
// channel.rs:342-366): the same seed, the same xorshift stream in the same order, so the ion's
// generator state and its RF / AC phases are the FP64 injection's bit for bit; the transforms of
// the draws (sqrt, log, sin / cos) run in FP32, as the reference's GPU path consumes FP32 ion
// states (its injection runs on the host, channel.rs:342-366, and is narrowed to f32 for the
// device). Positions take their FP32 offset from the axis in FP64, so they keep the axis exactly.
// GB300's FP64 pipe makes the FP64 transforms (about 360 FP64 operations per ion) the whole cost
// of the FP64 kernel k_inject; here an ion costs a few dozen FP32 operations.
__device__ __forceinline__ uint64_t xs_raw(uint64_t* st) {   // xorshift64 step, world.rs:386-392
    uint64_t x = *st;
    x ^= x << 13;
    x ^= x >> 7;
    x ^= x << 17;
    *st = x;
    return x;
}
// (x >> 11) / 2^53 as FP32: top 24 bits plus the next 29 scaled below them (within 1 ulp)
__device__ __forceinline__ float u53f(uint64_t x) {
    return fmaf((float)((uint32_t)(x >> 11) & 0x1FFFFFFFu), 0x1.0p-53f, (float)(uint32_t)(x >> 40) * 0x1.0p-24f);
}
__device__ __forceinline__ double u53d(uint64_t x) { return (double)(x >> 11) * 0x1.0p-53; }   // exact
// -ln u for u = (x >> 11) / 2^53 > 0, to FP32 accuracy also near u = 1, where 1 - u is formed
// exactly in integers and the logarithm taken as log1p(-(1 - u))
__device__ __forceinline__ float neg_log_u(uint64_t x) {
    const uint64_t k = x >> 11;
    if (k >= (1ull << 52)) return -log1pf(-(float)((1ull << 53) - k) * 0x1.0p-53f);
    return -logf(u53f(x));
}
// sqrt(-2 ln max(u, 1e-300)): the FP64 clamp lies below FP32's range; only u = 0 reaches it
__device__ __forceinline__ float gauss_radius(uint64_t x) {
    return (x >> 11) ? sqrtf(2.0f * neg_log_u(x)) : 37.1692219f;
}

__global__ void __launch_bounds__(128) k_inject_mixed(mqp::Batch b, mqd::JobTable jt, DevIons io, uint32_t n) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    uint32_t lo = 0, hi = jt.njobs;   // the job of ion i: last job with first <= i
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) >> 1;
        if (jt.first[mid] <= i) lo = mid; else hi = mid;
    }
    const mqp::JobC& j = jt.jc[lo];
    uint64_t st = mqp::splitmix(jt.seed[lo] + ((uint64_t)i - jt.first[lo]) * 0x9E37ull) | 1ull;
    float ox, oy, v0, v1, v2;
    if (b.launch == 1) {               // legacy launch, channel.rs:350-355
        const float kin = 0.1f * (0.75f + 0.75f * u53f(xs_raw(&st))) * (float)j.zc;
        const float vin = sqrtf(2.0f * kin * ((float)mqp::QE / (float)j.m));
        const float ang = (-10.0f + 20.0f * u53f(xs_raw(&st))) * (3.14159265f / 180.0f);
        float sa, ca;
        sincosf(ang, &sa, &ca);
        ox = oy = 0.0f;
        v0 = v1 = 0.707f * vin * sa;
        v2 = vin * ca;
    } else {
        if (b.launch == 2) {           // Gaussian spot
            const float r0 = gauss_radius(xs_raw(&st));
            const float c0 = cospif(2.0f * u53f(xs_raw(&st)));
            const float r1 = gauss_radius(xs_raw(&st));
            const float c1 = cospif(2.0f * u53f(xs_raw(&st)));
            ox = (float)b.sigma * r0 * c0;
            oy = (float)b.sigma * r1 * c1;
        } else {                       // uniform disc
            const float r = (float)b.r_inject * sqrtf(u53f(xs_raw(&st)));
            float sn, cs;
            sincospif(2.0f * u53f(xs_raw(&st)), &sn, &cs);
            ox = r * cs;
            oy = r * sn;
        }
        const float s_ion = (float)j.s_ion;
        const float ra = gauss_radius(xs_raw(&st));
        const float ca = cospif(2.0f * u53f(xs_raw(&st)));
        const float rb = gauss_radius(xs_raw(&st));
        const float cb = cospif(2.0f * u53f(xs_raw(&st)));
        v0 = s_ion * ra * ca;
        v1 = s_ion * rb * cb;
        v2 = s_ion * gauss_radius(xs_raw(&st));
    }
    const double ph_ac = u53d(xs_raw(&st));
    const double prf = u53d(xs_raw(&st));
    const uint64_t xf = xs_raw(&st);
    // first free path -ln max(u, 1e-7) * mfp / 10 (channel.rs:365-366) as a step count; u < 1e-7
    // exactly when (x >> 11) <= 900719925
    const float nl = (xf >> 11) <= 900719925ull ? 16.1180957f : neg_log_u(xf);
    const float first = nl * (float)j.mfp_mean / 10.0f;
    const float vmag = sqrtf(fmaf(v0, v0, fmaf(v1, v1, v2 * v2)));
    const float s0 = floorf(first / vmag / (float)b.dt) + 1.0f;
    io.x[i] = b.a + (double)ox; io.y[i] = b.a + (double)oy; io.z[i] = b.z_inject;
    io.vx[i] = (double)v0; io.vy[i] = (double)v1; io.vz[i] = (double)v2;
    io.ph_rf[i] = b.rf_phase0 ? 0.0 : prf; io.ph_ac[i] = ph_ac;
    io.rng[i] = st | 1ull;
    io.leg[i] = s0 < 2147483520.0f ? (int32_t)s0 : 2147483647;
    io.steps[i] = 0; io.ncoll[i] = 0; io.status[i] = 0; io.jid[i] = lo;
}

// initial live list (ions with status 0, warp-ballot compaction) and their working state: the
// FP64 position / velocity in grid units as double-floats and the phase offsets as fixed-point
// turns, converted here with every lane of a warp busy instead of one lane at a time in k_mixed
__global__ void k_init_list(DevIons io, uint32_t n, uint32_t* list, Ctrs* ctr, MixBatch B, float* __restrict__ keep,
                            uint64_t* __restrict__ kph, uint8_t* __restrict__ staged) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    const bool live = i < n && io.status[i] == 0;
    if (i < n) staged[i] = live ? 1 : 0;
    if (live) {
        const double gx[3] = {io.x[i] * B.inv_h, io.y[i] * B.inv_h, io.z[i] * B.inv_h};
        const double gu[3] = {io.vx[i] * B.v2u, io.vy[i] * B.v2u, io.vz[i] * B.v2u};
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const float xh = (float)gx[d], uh = (float)gu[d];
            keep[(size_t)(0 + d) * n + i] = xh; keep[(size_t)(3 + d) * n + i] = (float)(gx[d] - (double)xh);
            keep[(size_t)(6 + d) * n + i] = uh; keep[(size_t)(9 + d) * n + i] = (float)(gu[d] - (double)uh);
        }
        kph[i] = (uint64_t)(io.ph_rf[i] * 0x1.0p63) << 1;
        kph[(size_t)n + i] = (uint64_t)(io.ph_ac[i] * 0x1.0p63) << 1;
    }
    const unsigned m = __ballot_sync(FULL, live);
    const uint32_t lane = threadIdx.x & 31;
    if (m) {
        const int leader = __ffs(m) - 1;
        uint32_t base = 0;
        if ((int)lane == leader) base = atomicAdd(&ctr->count[0], (uint32_t)__popc(m));
        base = __shfl_sync(FULL, base, leader);
        if (live) list[base + __popc(m & ((1u << lane) - 1u))] = i;
    }
}

// FP64 position and velocity of every ion staged at the start of the call, from its working state
__global__ void k_unstage(DevIons io, uint32_t n, MixBatch B, const float* __restrict__ keep,
                          const uint8_t* __restrict__ staged) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n || !staged[i]) return;
    double* const xs[3] = {io.x, io.y, io.z};
    double* const vs[3] = {io.vx, io.vy, io.vz};
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        xs[d][i] = ((double)keep[(size_t)(0 + d) * n + i] + (double)keep[(size_t)(3 + d) * n + i]) * B.h;
        vs[d][i] = ((double)keep[(size_t)(6 + d) * n + i] + (double)keep[(size_t)(9 + d) * n + i]) * B.u2v;
    }
}

// ---------------------------------------------------------------- cell order of the live list
// Before a launch, the live list can be put in the Morton order of the ions' cells (a counting sort
// on the top bits of the 30-bit code), so the 32 lanes of a warp, which take consecutive queue
// slots, start in neighbouring cells and share cache lines in their cell gathers.  Order within a
// bin is the atomics' arrival order: per-ion results do not depend on the order.
// Bits 0..9 of v spread to every third bit (the "part 1 by 2" step of Morton encoding).
__device__ __forceinline__ uint32_t spread10(uint32_t v) {
    v &= 0x3ffu;
    v = (v ^ (v << 16)) & 0xff0000ffu;
    v = (v ^ (v << 8)) & 0x0300f00fu;
    v = (v ^ (v << 4)) & 0x030c30c3u;
    v = (v ^ (v << 2)) & 0x09249249u;
    return v;
}

constexpr int kScanBlock = 1024;          // threads of the scan kernels
constexpr int kScanItems = 4;             // bins per scan thread
constexpr uint32_t kScanTile = kScanBlock * kScanItems;

// bin of every listed ion (cell Morton code >> shift) and the bins' counts; lanes of a warp with the
// same bin add to it with one atomic (ions cluster in few cells, e.g. right after injection)
__global__ void k_sort_keys(const uint32_t* __restrict__ list, const Ctrs* __restrict__ ctr, int slot,
                            const float* __restrict__ keep, uint32_t n_all, MixBatch B, uint32_t shift,
                            uint32_t* __restrict__ keys, uint32_t* __restrict__ bins) {
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= ctr->count[slot]) return;
    const uint32_t id = list[t];
    const uint32_t ci = (uint32_t)clampi(__float2int_rd(keep[(size_t)0 * n_all + id]), 0, B.nx - 2);
    const uint32_t cj = (uint32_t)clampi(__float2int_rd(keep[(size_t)1 * n_all + id]), 0, B.ny - 2);
    const uint32_t ck = (uint32_t)clampi(__float2int_rd(keep[(size_t)2 * n_all + id]), 0, B.nz - 2);
    const uint32_t key = (spread10(ci) | (spread10(cj) << 1) | (spread10(ck) << 2)) >> shift;
    keys[t] = key;
    const unsigned peers = __match_any_sync(__activemask(), key);
    if ((threadIdx.x & 31) == (unsigned)(__ffs(peers) - 1)) atomicAdd(bins + key, (uint32_t)__popc(peers));
}

// exclusive scan of a tile of kScanTile counts in place; the tile's total to sums[blockIdx.x]
__global__ void __launch_bounds__(kScanBlock) k_scan_tiles(uint32_t* __restrict__ v, uint32_t n, uint32_t* __restrict__ sums) {
    __shared__ uint32_t warp_tot[kScanBlock / 32];
    const uint32_t base = blockIdx.x * kScanTile + threadIdx.x * kScanItems;
    uint32_t x[kScanItems], run = 0;
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        x[k] = base + k < n ? v[base + k] : 0u;
        run += x[k];
    }
    const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    uint32_t inc = run;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(FULL, inc, o);
        if (lane >= (uint32_t)o) inc += y;
    }
    if (lane == 31) warp_tot[w] = inc;
    __syncthreads();
    if (w == 0) {
        uint32_t t = warp_tot[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(FULL, t, o);
            if (lane >= (uint32_t)o) t += y;
        }
        warp_tot[lane] = t;   // inclusive over warps
    }
    __syncthreads();
    uint32_t off = inc - run + (w ? warp_tot[w - 1] : 0u);
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        if (base + k < n) v[base + k] = off;
        off += x[k];
    }
    if (threadIdx.x == kScanBlock - 1) sums[blockIdx.x] = warp_tot[kScanBlock / 32 - 1];
}

// add the scanned tile totals to every tile
__global__ void k_scan_add(uint32_t* __restrict__ v, uint32_t n, const uint32_t* __restrict__ sums) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) v[i] += sums[i / kScanTile];
}

// every listed ion to the next free place of its bin (one atomic per bin per warp)
__global__ void k_sort_scatter(const uint32_t* __restrict__ list, const Ctrs* __restrict__ ctr, int slot,
                               const uint32_t* __restrict__ keys, uint32_t* __restrict__ bins, uint32_t* __restrict__ out) {
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= ctr->count[slot]) return;
    const uint32_t key = keys[t], lane = threadIdx.x & 31;
    const unsigned peers = __match_any_sync(__activemask(), key);
    const int leader = __ffs(peers) - 1;
    uint32_t base = 0;
    if ((int)lane == leader) base = atomicAdd(bins + key, (uint32_t)__popc(peers));
    base = __shfl_sync(peers, base, leader);
    out[base + __popc(peers & ((1u << lane) - 1u))] = list[t];
}

// prepare launch: clear the queue head and the output count, and add the launch's queue length
__global__ void k_prep(Ctrs* ctr, int out_slot) {
    ctr->head = 0;
    for (int k = 0; k < kMaxLegs; ++k) ctr->head_g[k] = ctr->handed[k] = 0;
    ctr->handed[kMaxLegs] = 0;
    ctr->count[out_slot] = 0;
    ctr->open = ctr->count[out_slot ^ 1];
    ctr->queued += ctr->count[out_slot ^ 1];
}

void split(double v, float& h, float& l) {
    h = (float)v;
    l = (float)(v - (double)h);
}

uint64_t fix64(double turns_per_step) {   // round(frac(w) * 2^64)
    double f = turns_per_step - floor(turns_per_step);
    long double s = (long double)f * 18446744073709551616.0L;
    long double r = floorl(s + 0.5L);
    if (r >= 18446744073709551616.0L) return 0;
    return (uint64_t)r;
}

}  // namespace

cudaError_t launch_inject(const mqp::Batch& b, mqd::JobTable jt, DevIons io, uint32_t n, cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    k_inject_mixed<<<(n + 127) / 128, 128, 0, st>>>(b, jt, io, n);
    return cudaGetLastError();
}

MixJob make_mix_job(const mqp::JobC& j, const mqp::Batch& b) {
    MixJob m;
    std::memset(&m, 0, sizeof(m));
    m.kick = (float)(j.qmdt * b.dt / b.h);
    m.v_ac = (float)j.v_ac;
    m.cand_a = (float)(j.nsd * b.h / b.dt);
    m.cand_b = (float)(j.nsd * 1.5957691216057308 * j.s_gas);   // n sigma dt E|V| (thermal_partner)
    m.s_gas = (float)j.s_gas;
    m.mr = (float)j.mr;
    m.floor_v = (float)j.floor_v;
    m.mfp_mean = (float)j.mfp_mean;
    uint64_t w = fix64(j.w_ac);
    m.w_ac_lo = (uint32_t)w;
    m.w_ac_hi = (uint32_t)(w >> 32);
    double s, c;
    mqp::sincos2pi(j.w_ac, &s, &c);
    m.cw_ac = (float)c;
    m.sw_ac = (float)s;
    m.use_ac = j.use_ac;
    return m;
}

MixBatch make_mix_batch(const mqp::Batch& b) {
    MixBatch m;
    std::memset(&m, 0, sizeof(m));
    m.h = b.h;
    m.inv_h = 1.0 / b.h;
    m.dt = b.dt;
    m.u2v = b.h / b.dt;
    m.v2u = b.dt / b.h;
    m.v_rf = (float)b.v_rf;
    m.dt_f = (float)b.dt;
    m.u2v_f = (float)m.u2v;
    m.v2u_f = (float)m.v2u;
    uint64_t w = fix64(b.w_rf);
    m.w_rf_lo = (uint32_t)w;
    m.w_rf_hi = (uint32_t)(w >> 32);
    double s, c;
    mqp::sincos2pi(b.w_rf, &s, &c);
    m.cw_rf = (float)c;
    m.sw_rf = (float)s;
    split(b.z_exit / b.h, m.z_exit_h, m.z_exit_l);
    split(b.z_return / b.h, m.z_ret_h, m.z_ret_l);
    split(b.crash_z0 / b.h, m.cz0_h, m.cz0_l);
    split(b.crash_z1 / b.h, m.cz1_h, m.cz1_l);
    // a plane farther than this cannot be crossed whatever the low part holds (below half an ulp of z)
    const float near = fmaxf(0x1.0p-6f, (float)b.nz * 0x1.0p-20f);
    m.z_exit_near = m.z_exit_h - near;
    m.z_ret_near = m.z_ret_h + near;
    m.lim_x = (float)(b.nx - 1);
    m.lim_y = (float)(b.ny - 1);
    m.lim_z = (float)(b.nz - 1);
    m.nx = b.nx; m.ny = b.ny; m.nz = b.nz;
    m.nearest = b.nearest;
    m.legacy_coll = b.legacy_coll;
    m.max_steps = b.max_steps;
    return m;
}

Tuning default_tuning(int device, size_t nodes) {
    Tuning t;
    int sms = 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) { cudaGetLastError(); sms = 1; }
    t.sms = sms;
    // Record width and, with resident_blocks(), ions in flight per SM by the size of the grid (bytes of its 48-byte records). Wide records
    // win while the part that the ions see lies in L2, with 3 blocks per SM and near the end with 2; then
    // narrow ones with 2 blocks, until the gathers of fewer ions in flight hit the caches so much more often that
    // 1 is better. Batch of 512,000 ions, ms, wide 3 / wide 2 / narrow 2 / narrow 1: 0.30 GB (0.100 mm channel) 10.7 / 12.0 /
    // 13.3 / 18.5, 0.40 GB 11.3 / 12.1 / 13.4 / -, 0.45 GB 14.7 / 12.4 / 14.0 / -, 0.51 GB 17.6 / 12.8 / 14.3 / -, 0.58 GB
    // 20.6 / - / 14.5 / 19.9, 1.22 GB 31.5 / - / 15.4 / 20.6, 2.6 GB - / - / 19.4 / 23.0, 3.4 GB - / - / 24.2 / 24.6,
    // 4.6 GB - / - / 28.9 / 25.9, 8.0 GB - / - / 35.7 / 28.2.
    const double rec = 48.0 * (double)nodes;
    t.wide = rec < 0.55e9 ? 1 : 0;
    t.blocks_per_sm = rec < 0.42e9 ? 3 : rec < 0.55e9 ? 2 : 1;
    return t;
}

// Ions that the lane groups hold at once: a list of up to so many is stepped by them alone, a longer
// one's last so many are handed to them.
static uint32_t hand_entries(int sms, bool nearest) { return (uint32_t)sms * (uint32_t)(group_block(nearest) / 4); }
uint32_t group_ions(const Tuning& t, bool nearest) { return hand_entries(t.sms, nearest); }

// Steps of the lane-group launches of one round of `chunk` steps. Between them the ions that are left are
// spread over full warps again: worth its 10 us where warps hold many ions each and these end one by one
// over many thousand steps, as with legacy collisions (Fig. 4 scan of 26,000 ions: 11.9 -> 10.7 ms). Thermal
// ions end early or not at all (S14 sweep 39.2 against 39.8 ms with such legs), and where a warp has
// one or two ions there is nothing to pack.
static int plan_legs(uint32_t chunk, bool many_legs, uint32_t legs[kMaxLegs]) {
    uint32_t leg = many_legs ? 1024u : chunk, left = chunk;
    int k = 0;
    while (left > 0) {
        legs[k] = k == kMaxLegs - 1 || left < leg + leg / 2 ? left : leg;
        left -= legs[k++];
        leg += leg / 2;
    }
    return k;
}

void release(Scratch& s) {
    if (s.graph) cudaGraphExecDestroy(s.graph);
    for (void* p : {s.lists, s.ctrs, s.params, s.jobs, s.nodes, s.keep, s.sort}) if (p) cudaFree(p);
    for (auto& e : s.ev) if (e) cudaEventDestroy(e);
    s = Scratch();
}

// the stepping kernel for the batch's physics and the tuning (the nearest-node field mode reads one
// record per fill, so the L1 prefetch of the next cell does not apply to it)
typedef decltype(&k_mixed<true, true, true, false, 3>) Kernel;
static Kernel pick_kernel(const Tuning& t, bool legacy, bool nearest, int blocks) {
    if (nearest) {
        if (legacy) return t.wide ? k_mixed<true, false, true, true, 5> : k_mixed<true, false, false, true, 5>;
        return t.wide ? k_mixed<false, false, true, true, 5> : k_mixed<false, false, false, true, 5>;
    }
    if (t.wide && blocks == 4) {
        if (legacy) return t.prefetch ? k_mixed<true, true, true, false, 4> : k_mixed<true, false, true, false, 4>;
        return t.prefetch ? k_mixed<false, true, true, false, 4> : k_mixed<false, false, true, false, 4>;
    }
    if (legacy) {
        if (t.wide) return t.prefetch ? k_mixed<true, true, true, false, 3> : k_mixed<true, false, true, false, 3>;
        if (blocks == 3) return t.prefetch ? k_mixed<true, true, false, false, 3> : k_mixed<true, false, false, false, 3>;
        return t.prefetch ? k_mixed<true, true, false, false, 2> : k_mixed<true, false, false, false, 2>;
    }
    if (t.wide) return t.prefetch ? k_mixed<false, true, true, false, 3> : k_mixed<false, false, true, false, 3>;
    return t.prefetch ? k_mixed<false, true, false, false, 2> : k_mixed<false, false, false, false, 2>;
}

int resident_blocks(const Tuning& t, size_t nodes, size_t n, bool legacy, bool nearest) {
    if (nearest) {   // no 8-corner cache (about 96 registers instead of 167): as many blocks as fit
        int nb = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, pick_kernel(t, legacy, true, 0), t.tpb, 0) == cudaSuccess && nb > 0) return nb;
        cudaGetLastError();
        return t.blocks_per_sm;
    }
    // What the narrow kernels' registers leave room for: three with legacy collisions, cut to 168 registers without spills, two
    // with thermal ones. Three are worth it on small grids for more ions than two hold: legacy collisions, 3,000 steps at 2 / 3
    // blocks, 0.100 mm 30,000 ions 3.6 / 4.1 ms, 40,000 4.9 / 4.2, 80,000 8.6 / 7.9, 400,000 38.8 / 32.3; 0.050 mm 400,000 52.5 / 54.2.
    const int narrow = legacy ? 3 : 2;
    if (!t.auto_blocks) return t.wide || t.blocks_per_sm < narrow ? t.blocks_per_sm : narrow;
    if (!t.wide && legacy && t.blocks_per_sm == 3 && n > 256 * (size_t)t.sms) return 3;
    if (!t.wide) return 48.0 * (double)nodes < 3.5e9 ? 2 : 1;   // default_tuning has the figures
    // three with wide records are four for a list of eight or more ions a lane, which outlasts its uneven end:
    // 1,280,000 ions 22.1 -> 21.1 ms, 640,000 13.6 -> 13.2, 320,000 the same, 62,000 (S14 sweep) 39.0 -> 40.4
    return t.blocks_per_sm == 3 && n > 2048 * (size_t)t.sms ? 4 : t.blocks_per_sm;
}

typedef decltype(&k_mixed_group<true, true, false>) GroupKernel;
static GroupKernel pick_group_kernel(const Tuning& t, const MixBatch& mb) {
    if (mb.nearest) {
        if (mb.legacy_coll) return t.wide ? k_mixed_group<true, true, true> : k_mixed_group<true, false, true>;
        return t.wide ? k_mixed_group<false, true, true> : k_mixed_group<false, false, true>;
    }
    if (mb.legacy_coll) return t.wide ? k_mixed_group<true, true, false> : k_mixed_group<true, false, false>;
    return t.wide ? k_mixed_group<false, true, false> : k_mixed_group<false, false, false>;
}

// bins of the cell sort: the top min(22, 3 b) bits of the Morton code, b the bits of the largest
// cell index (nbins <= 2^22, so the tile totals fit one scan tile)
struct SortPlan {
    uint32_t nbins, tiles, shift;
};
static SortPlan sort_plan(const MixBatch& mb, uint32_t n) {
    (void)n;
    int32_t mx = mb.nx > mb.ny ? mb.nx : mb.ny;
    mx = mx > mb.nz ? mx : mb.nz;
    uint32_t bits = 1;
    while ((1u << bits) < (uint32_t)(mx - 1)) ++bits;   // cell indices 0 .. mx - 2
    const uint32_t code = 3 * bits, kb = code < 22 ? code : 22;
    SortPlan p;
    p.nbins = 1u << kb;
    p.tiles = (p.nbins + kScanTile - 1) / kScanTile;
    p.shift = code - kb;
    return p;
}
static size_t sort_bytes(const MixBatch& mb, uint32_t n) {
    const SortPlan p = sort_plan(mb, n);
    return sizeof(uint32_t) * ((size_t)p.nbins + p.tiles + 1 + 2 * (size_t)n);
}

static cudaError_t enqueue_launches(const Scratch& s, const Tuning& t, int blocks_per_sm, const MixBatch& mb, DevIons io,
                                    uint32_t n, uint32_t launches, uint32_t chunk, uint32_t last_chunk, cudaStream_t st,
                                    uint32_t* kernels) {
    uint32_t* lists = static_cast<uint32_t*>(s.lists);
    Ctrs* ctr = static_cast<Ctrs*>(s.ctrs);
    const MixJob* jobs = static_cast<const MixJob*>(s.jobs);
    const float4* nodes = static_cast<const float4*>(s.nodes);
    uint64_t* kph = static_cast<uint64_t*>(s.keep);
    float* keep = reinterpret_cast<float*>(kph + (size_t)2 * n);
    const int grid = t.sms * blocks_per_sm;
    const SortPlan sp = sort_plan(mb, n);
    uint32_t* bins = static_cast<uint32_t*>(s.sort);
    uint32_t* sums = bins + sp.nbins;
    uint32_t* keys = sums + sp.tiles + 1;
    uint32_t* sorted = keys + n;
    for (uint32_t L = 0; L < launches; ++L) {
        const int in = (int)(L & 1);
        k_prep<<<1, 1, 0, st>>>(ctr, in ^ 1);
        const uint32_t ch = (L + 1 == launches) ? last_chunk : chunk;
        const uint32_t* li = lists + (size_t)in * n;
        uint32_t* lo = lists + (size_t)(in ^ 1) * n;
        if (t.sort_cells) {   // this launch's list in the cells' Morton order
            cudaMemsetAsync(bins, 0, (size_t)sp.nbins * sizeof(uint32_t), st);
            const unsigned gi = (n + 255) / 256;
            k_sort_keys<<<gi, 256, 0, st>>>(li, ctr, in, keep, n, mb, sp.shift, keys, bins);
            k_scan_tiles<<<sp.tiles, kScanBlock, 0, st>>>(bins, sp.nbins, sums);
            k_scan_tiles<<<1, kScanBlock, 0, st>>>(sums, sp.tiles, sums + sp.tiles);   // tiles <= kScanTile
            k_scan_add<<<(sp.nbins + 255) / 256, 256, 0, st>>>(bins, sp.nbins, sums);
            k_sort_scatter<<<gi, 256, 0, st>>>(li, ctr, in, keys, bins, sorted);
            li = sorted;
            *kernels += 5;
        }
        const Kernel kern = pick_kernel(t, mb.legacy_coll != 0, mb.nearest != 0, blocks_per_sm);
        const uint32_t hand_at = hand_entries(t.sms, mb.nearest != 0);
        uint2* hand = reinterpret_cast<uint2*>(ctr + 1);
        if (n > hand_at) {
            kern<<<grid, t.tpb, 0, st>>>(nodes, mb, jobs, io, li, lo, ctr, in, ch, keep, kph, n, hand, hand_at);
            *kernels += 1;
        }
        const int sm = group_block(mb.nearest != 0) / 4 * group_floats(mb.legacy_coll != 0) * (int)sizeof(float);
        const GroupKernel gk = pick_group_kernel(t, mb);
        cudaFuncSetAttribute(gk, cudaFuncAttributeMaxDynamicSharedMemorySize, sm);
        uint32_t legs[kMaxLegs];
        const int nlegs = plan_legs(ch, mb.legacy_coll && L == 0 && n > 2u * kGroupFirst * (uint32_t)t.sms, legs);
        for (int k = 0; k < nlegs; ++k)
            gk<<<t.sms, group_block(mb.nearest != 0), sm, st>>>(nodes, mb, jobs, io, li, hand, lo, ctr, in, ch, k, legs[k], keep, kph, n, hand_at);
        *kernels += 1u + (uint32_t)nlegs;
    }
    return cudaGetLastError();
}

cudaError_t pack_nodes(Scratch& s, DevGrid g, uint64_t grid_gen, int wide, cudaStream_t st, uint32_t* kernels) {
    const int stride = wide ? 6 : 3;
    if (s.nodes && s.nodes_gen == grid_gen && s.nodes_stride == stride) return cudaSuccess;
    cudaError_t e;
    const size_t n = (size_t)g.nx * g.ny * g.nz;
    const size_t bytes = (size_t)stride * n * sizeof(float4);
    if (s.nodes_cap < bytes) {
        if (s.nodes) cudaFree(s.nodes);
        s.nodes = nullptr; s.nodes_cap = 0;
        if ((e = cudaMalloc(&s.nodes, bytes)) != cudaSuccess) return e;
        s.nodes_cap = bytes;
    }
    k_pack_nodes<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(g.rf, g.dc, g.ac, static_cast<float4*>(s.nodes), n, g.nx, g.ny, g.nz,
                                                              stride);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    *kernels += 1;
    s.nodes_gen = grid_gen;
    s.nodes_stride = stride;
    return cudaSuccess;
}

cudaError_t run(Scratch& s, const Tuning& t, DevGrid g, uint64_t grid_gen, const mqp::Batch& b, const MixJob* jobs,
                size_t njobs, DevIons io, uint32_t n, uint32_t max_more, int write_states, cudaStream_t st, RunInfo* info) {
    cudaError_t e;
    *info = RunInfo();
    if (n == 0) return cudaSuccess;
    if (t.tpb != 128) return cudaErrorInvalidValue;   // the kernel is compiled for 128-thread blocks
    if ((e = pack_nodes(s, g, grid_gen, t.wide, st, &info->kernel_launches)) != cudaSuccess) return e;
    const size_t list_bytes = (size_t)2 * n * sizeof(uint32_t);
    if (s.list_cap < list_bytes) {
        if (s.lists) cudaFree(s.lists);
        s.lists = nullptr; s.list_cap = 0;
        if ((e = cudaMalloc(&s.lists, list_bytes)) != cudaSuccess) return e;
        s.list_cap = list_bytes;
    }
    if (!s.ctrs && (e = cudaMalloc(&s.ctrs, sizeof(Ctrs) + sizeof(uint2) * 2 * (size_t)hand_entries(t.sms, true))) != cudaSuccess) return e;
    if (s.jobs_cap < njobs * sizeof(MixJob)) {
        if (s.jobs) cudaFree(s.jobs);
        s.jobs = nullptr; s.jobs_cap = 0;
        if ((e = cudaMalloc(&s.jobs, njobs * sizeof(MixJob))) != cudaSuccess) return e;
        s.jobs_cap = njobs * sizeof(MixJob);
    }
    if (!s.ev[0]) { cudaEventCreate(&s.ev[0]); cudaEventCreate(&s.ev[1]); }
    if ((e = cudaMemcpyAsync(s.jobs, jobs, njobs * sizeof(MixJob), cudaMemcpyHostToDevice, st)) != cudaSuccess) return e;
    const MixBatch mb = make_mix_batch(b);
    // launches needed: every live ion has at most min(max_more, max_steps) steps left
    const uint64_t need = max_more < b.max_steps ? (uint64_t)max_more : (uint64_t)b.max_steps;
    if (need == 0) return cudaSuccess;
    const uint32_t chunk = t.chunk ? t.chunk : 4096;
    const uint32_t full = (uint32_t)((need + chunk - 1) / chunk);
    const uint32_t launches = (t.max_launches && t.max_launches < full) ? t.max_launches : full;
    const uint32_t last_chunk = launches < full ? chunk : (uint32_t)(need - (uint64_t)(launches - 1) * chunk);
    // working state: phase offsets (2 x u64), position / velocity double-floats (12 x f32) and the
    // staged flag (u8) of every ion
    const size_t keep_bytes = (size_t)n * (2 * sizeof(uint64_t) + 12 * sizeof(float) + 1);
    if (s.keep_cap < keep_bytes) {
        if (s.keep) cudaFree(s.keep);
        s.keep = nullptr; s.keep_cap = 0;
        if ((e = cudaMalloc(&s.keep, keep_bytes)) != cudaSuccess) return e;
        s.keep_cap = keep_bytes;
    }
    if (t.sort_cells && s.sort_cap < sort_bytes(mb, n)) {
        if (s.sort) cudaFree(s.sort);
        s.sort = nullptr; s.sort_cap = 0;
        if ((e = cudaMalloc(&s.sort, sort_bytes(mb, n))) != cudaSuccess) return e;
        s.sort_cap = sort_bytes(mb, n);
    }
    Ctrs* ctr = static_cast<Ctrs*>(s.ctrs);
    if ((e = cudaMemsetAsync(ctr, 0, sizeof(Ctrs), st)) != cudaSuccess) return e;
    uint64_t* kph = static_cast<uint64_t*>(s.keep);
    float* keep = reinterpret_cast<float*>(kph + (size_t)2 * n);
    uint8_t* staged = reinterpret_cast<uint8_t*>(keep + (size_t)12 * n);
    k_init_list<<<(n + 255) / 256, 256, 0, st>>>(io, n, static_cast<uint32_t*>(s.lists), ctr, mb, keep, kph, staged);
    info->kernel_launches += 1;
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    const int blocks = resident_blocks(t, (size_t)mb.nx * mb.ny * mb.nz, n, mb.legacy_coll != 0, mb.nearest != 0);
    cudaEventRecord(s.ev[0], st);
    uint32_t kernels = 0;
    const bool graph = t.use_graph && launches > 1;
    if (graph) {
        const uint64_t key[6] = {(uint64_t)(uintptr_t)s.lists, (uint64_t)n, launches, ((uint64_t)chunk << 32) | last_chunk,
                                 (uint64_t)(uintptr_t)io.x ^ ((uint64_t)blocks << 56) ^ ((uint64_t)t.prefetch << 60) ^
                                     ((uint64_t)t.wide << 61) ^ ((uint64_t)t.sort_cells << 63),
                                 (uint64_t)(uintptr_t)s.nodes ^ ((uint64_t)mb.legacy_coll << 62) ^ ((uint64_t)mb.nearest << 61)};
        cudaGraph_t gr = nullptr;
        if ((e = cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal)) != cudaSuccess) return e;
        enqueue_launches(s, t, blocks, mb, io, n, launches, chunk, last_chunk, st, &kernels);
        e = cudaStreamEndCapture(st, &gr);
        if (e != cudaSuccess) { if (gr) cudaGraphDestroy(gr); return e; }
        // re-use the instantiated graph when only kernel parameters changed
        bool updated = false;
        if (s.graph && std::memcmp(key, s.graph_key, sizeof(key)) == 0) {
            cudaGraphExecUpdateResultInfo ri;
            if (cudaGraphExecUpdate(s.graph, gr, &ri) == cudaSuccess) updated = true;
            else cudaGetLastError();
        }
        if (!updated) {
            if (s.graph) { cudaGraphExecDestroy(s.graph); s.graph = nullptr; }
            if ((e = cudaGraphInstantiate(&s.graph, gr, 0)) != cudaSuccess) { cudaGraphDestroy(gr); return e; }
            std::memcpy(s.graph_key, key, sizeof(key));
        }
        cudaGraphDestroy(gr);
        if ((e = cudaGraphLaunch(s.graph, st)) != cudaSuccess) return e;
        info->graph_replays = 1;
    } else {
        if ((e = enqueue_launches(s, t, blocks, mb, io, n, launches, chunk, last_chunk, st, &kernels)) != cudaSuccess) return e;
    }
    cudaEventRecord(s.ev[1], st);
    if (write_states) {
        k_unstage<<<(n + 255) / 256, 256, 0, st>>>(io, n, mb, keep, staged);
        info->kernel_launches += 1;
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
    }
    Ctrs h;
    if ((e = cudaMemcpyAsync(&h, ctr, sizeof(Ctrs), cudaMemcpyDeviceToHost, st)) != cudaSuccess) return e;
    if ((e = cudaStreamSynchronize(st)) != cudaSuccess) return e;
    cudaEventElapsedTime(&info->step_ms, s.ev[0], s.ev[1]);
    info->ion_steps = h.steps;
    info->cell_loads = h.cell_loads;
    info->ions_queued = h.queued;
    info->step_launches = launches;
    info->kernel_launches += kernels;
    // after the last launch the surviving list must be empty unless the step budget ran out
    const uint32_t survivors = h.count[launches & 1];
    info->survivors = survivors;
    info->watchdog = (survivors != 0 && max_more >= b.max_steps) ? 1 : 0;
    return cudaSuccess;
}

}  // namespace mqmix

MQ_CHECK_READER(mq_check_read_mixed)
