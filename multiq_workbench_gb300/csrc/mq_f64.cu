// Plain FP64 ion-trajectory kernel: a group of lanes per ion, FP64 state, f32 field nodes
// promoted to f64, global phase tables, xorshift64 collision Monte Carlo.  It evaluates
// exactly the operations of the FP64 CPU integrator in the same order and is compiled
// with --fmad=false, so its final states equal the CPU integrator's bit for bit.
//
// Reference: advance_with_field / fields_at / collide / is_crash
// (simulation/mqviz/src/world.rs:265-314,471-536) with chsim's switches
// (simulation/chsim/src/channel.metal:56-62,100-121; channel.rs:397-426).
//
// Also here: device injection (Ion::inject, world.rs:407-422), phase tables
// (Clock::fill, world.rs:445-465), the combined DC field (Fields::dc_field,
// channel.rs:220-226) and the per-job summary (summarize, channel.rs:496-506).
#include "mq_internal.h"
#include "mq_check.h"
#include "mq_f64dev.h"

#include <cmath>

namespace mqd {
namespace {

using mqp::Batch;
using mqp::JobC;
using namespace mqf;

__global__ void k_inject(Batch b, JobTable jt, DevIons io, uint32_t n) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    // job of ion i: last job with first <= i
    uint32_t lo = 0, hi = jt.njobs;   // invariant first[lo] <= i < first[hi]
    while (hi - lo > 1) {
        uint32_t mid = (lo + hi) >> 1;
        if (jt.first[mid] <= i) lo = mid; else hi = mid;
    }
    uint64_t q = (uint64_t)i - jt.first[lo];
    uint64_t seed = mqp::splitmix(jt.seed[lo] + q * 0x9E37ull);
    mqp::Ion0 o;
    mqp::inject_one(b, jt.jc[lo], seed, &o);
    io.x[i] = o.x[0]; io.y[i] = o.x[1]; io.z[i] = o.x[2];
    io.vx[i] = o.v[0]; io.vy[i] = o.v[1]; io.vz[i] = o.v[2];
    io.ph_rf[i] = o.ph_rf; io.ph_ac[i] = o.ph_ac; io.rng[i] = o.rng; io.leg[i] = o.leg;
    io.steps[i] = 0; io.ncoll[i] = 0; io.status[i] = 0; io.jid[i] = lo;
}

__global__ void k_phase_table(double w, uint32_t len, double2* out) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= len) return;
    double s, c;
    mqp::phase_at(w, i, &s, &c);
    out[i] = make_double2(s, c);
}

__device__ __forceinline__ void table_get(const double2* t, uint32_t tlen, double w, uint32_t n, double* s, double* c) {
    if (n < tlen) { double2 v = __ldg(t + n); *s = v.x; *c = v.y; }
    else mqp::phase_at(w, n, s, c);
}

// ---------------------------------------------------------------- the step kernel
// What bounds it: GB300's FP64 pipe. An SM takes one FP64 warp instruction per 19 cycles (a warp that
// has its scheduler's share to itself one per 64), however many lanes are active and however much
// independent work the warp has. A step is about 200 FP64 operations: with one lane per ion it took
// 9 us, and a warp lasted as long as its longest-lived ion, with 6 of 32 lanes active on average.
// Here a group of G lanes steps one ion, so that one instruction does several of its operations:
// each lane owns an axis (position, velocity, cell) and one of the eight cell corners (two for
// G = 4), whose weight and products with the nine field components it forms; the nine sums over the
// corners run side by side in nine lanes (G = 16) or three to a lane (G = 4), and the drive's
// products ride in idle lanes. 26 (G = 16) or 59 (G = 4) FP64 instructions a step remain, and
// groups take the next ion of a queue when theirs ends. Comparisons, conversions, corner reloads
// and the collision test (against an FP32 bound, exact only where that does not decide) stay off
// the pipe. Every operation is the CPU integrator's, in its order: results are its bits.
// Which G: 16 up to the ions that one warp per scheduler holds (f64_hand_entries), where latency is all
// that counts: 1.8 us a step for up to 1,216 ions against 3.4 with G = 4 (S14 grid, no gas). Above, the
// pipe is full and 4 lanes waste fewer slots: 4,864 ions 3.4 us, 58,368 ions 25 us a step. The last ions of
// a large call go on in groups of 16.
// Measured (whole run_batch calls, before -> now): mass scan of 25,000 ions 162 -> 32 ms; S14 point with
// 20,000 ions and up to 75,000 steps 1,098 -> 197 ms.
constexpr int kBlock = 256;            // 8 warps: two per scheduler, one to fill the other's gaps
constexpr int kPad = 120 * 1024;       // dynamic shared memory asked for: so much that no second block fits (57 KB are used)
constexpr uint32_t kPollSteps = 32;    // steps between looks at the count of open ions
constexpr uint32_t kLaneRound = 1024;  // steps of one launch of the one-lane kernel (thermal collisions an eighth of it: fewer ions last)

// Shared memory of a group, in doubles: the fractions of the three axes as pairs {1 - t, t}, the
// products of the nine sums (rows of 8 corners, 10 apart: 16-byte reads of the rows meet no bank
// twice), and what the lanes hand each other besides: nine weighted sums, four drive products and
// the drive amplitudes.
constexpr int kRow = 10;
constexpr int kSums = 6 + 9 * kRow;
constexpr int kGroupDoubles = kSums + 16;

template <int G>
__global__ void __launch_bounds__(kBlock, 1)
k_f64_step(DevGrid g, Batch b, const JobC* __restrict__ jobs, const double2* __restrict__ rf_tab,
           const double2* __restrict__ ac_tab, uint32_t tlen, DevIons io, uint32_t n, uint32_t max_more,
           F64Ctrs* __restrict__ ctr, uint2* hand, uint32_t hand_at, int from_hand) {
    constexpr int GPW = 32 / G;            // groups per warp
    constexpr int NC = G == 16 ? 1 : 2;    // corners per lane
    constexpr int NP = G == 16 ? 5 : 9;    // sums a lane has products of, per corner
    constexpr int NS = G == 16 ? 1 : 3;    // sums a lane adds up
    extern __shared__ __align__(16) double sm[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, gl = lane % G, base = lane - gl;
    const int d = gl % 3;                  // the lane's axis; lanes 0..2 own it
    double* const tw = sm + (size_t)(threadIdx.x / G) * kGroupDoubles;
    double* const prod = tw + 6;
    double* const xch = tw + kSums;
    const uint32_t count = from_hand ? ctr->handed : n;
    // ions handed to a later launch instead of being finished: once at most hand_at are open
    const bool hands = !from_hand && hand != nullptr;
    uint32_t* const head = from_hand ? &ctr->head_b : &ctr->head_a;
    // the first ions, spread so that every scheduler of every SM has work before any has two warps
    const uint32_t first = (uint32_t)((((warp >> 2) * GPW + lane / G) * 4 + (warp & 3)) * gridDim.x + blockIdx.x);
    const uint32_t groups = gridDim.x * (kBlock / 32) * GPW;

    const double h = g.h, inv_h = g.inv_h, dt = b.dt;
    const int32_t nd = d == 0 ? g.nx : d == 1 ? g.ny : g.nz;
    const long long lim_c = __double_as_longlong((double)(nd - 2));
    const size_t nx = (size_t)g.nx, ny = (size_t)g.ny;
    [[maybe_unused]] const size_t total = nx * ny * (size_t)g.nz;   // bounds-checked build
    // High words of the positions that no plane or face can end: strictly between the words of the
    // limits (positive doubles order like their words), so one compare per lane clears a step
    const int up = min(__double2hiint(b.lim[d]), d == 2 ? __double2hiint(b.z_exit) : 0x7fffffff);
    const int in_lo = d == 2 ? __double2hiint(b.z_return) + 1 : 0;
    const unsigned in_n = gl < 3 ? (unsigned)max(up - in_lo, 0) : 0xffffffffu;
    // the lane's corner (G = 4: that and the one with di = 1; corner c = 4 di + 2 dj + dk) and, for
    // G = 16, which products (lanes 0..7 sums 0..4, lanes 8..15 sums 5..8) and which sum it has
    // (sum 3 f + d of field f: RF, AC, DC; lanes 9..15 repeat sums 0..6 and keep nothing of it)
    const int cn = G == 16 ? gl & 7 : gl;
    const bool upper = G == 16 && gl >= 8;
    const int chain = G == 16 ? (gl < 9 ? gl : gl - 9) : gl % 3;
    // Drive amplitudes amp (sin cos0 + cos sin0) of RF and AC for the next step. G = 16: lanes 9..12
    // form the four products, sums and amplitudes in the instructions that the sums' lanes use for
    // theirs. G = 4: even lanes RF, odd lanes AC, lanes 2 and 3 the second product.
    const bool drives = G == 16 ? gl >= 9 : true;
    const bool is_ac = G == 16 ? gl >= 11 : (gl & 1) != 0;
    const bool second = G == 16 ? (gl == 10 || gl == 12) : (gl & 2) != 0;
    // where the lane's first two addends lie: {RF, AC} sums of its axis, or the two drive products
    const int i0 = G == 16 && gl >= 9 ? (gl >= 11 ? 11 : 9) : d, i1 = G == 16 && gl >= 9 ? i0 + 1 : d + 3;

    bool have = false, drained = false, fresh = true;
    uint32_t id = 0, age = 0, left = 1, ncoll = 0, jid = 0;
    int32_t leg = 0;
    uint64_t rng = 1;
    double x = 0.0, v = 0.0, cell = 0.0, kick = 0.0, ph = 0.0, w_tone = 0.0, coef = 0.0;
    float nsd2 = 0.0f, ub0 = 0.0f;
    int32_t ci = -1, cj = -1, ck = -1;
    uint32_t mask = 0;
    double val[NC][NP];
    const double2* tab = rf_tab;
    bool use_ac = false;
    double S = 0.0, Cc = 0.0;
#pragma unroll
    for (int k = 0; k < NC; ++k)
#pragma unroll
        for (int m = 0; m < NP; ++m) val[k][m] = 0.0;
    unsigned long long steps_total = 0;
    uint32_t live = 0;
    bool turn = true;   // some group of the warp has no ion

    // the cell of position x and its fractions t of it; refills the corner values of the groups in `upd`
    // that changed cell. A fraction in [0, 1) of the cell it had means that the cell is the same.
    auto refill = [&](bool upd, double gx) -> double {
        const int32_t ca = cell_lo_bits(gx, nd, lim_c);
        cell = i2d_bits(ca);
        const double t = gx - cell;
        const int32_t ni = __shfl_sync(FULL, ca, base), nj = __shfl_sync(FULL, ca, base + 1), nk = __shfl_sync(FULL, ca, base + 2);
        const bool move = upd && (ni != ci || nj != cj || nk != ck);
        bool c0 = false, c1 = false;
        if (move) {
            ci = ni; cj = nj; ck = nk;
            // every load is asked for before the first value is used
            float r[NC][9], solid[2] = {0.0f, 0.0f};
#pragma unroll
            for (int k = 0; k < NC; ++k) {
                const int di = G == 16 ? cn >> 2 : k;
                size_t q = (size_t)(ci + di) + nx * ((size_t)(cj + ((cn >> 1) & 1)) + ny * (size_t)(ck + (cn & 1)));
                q = MQ_CHK(q, total, MQ_SITE_F64_FIELD);
                const float4 a4 = __ldg(g.ac + q), o4 = __ldg((upper ? g.dc : g.rf) + q);
                if (G == 16) {
                    r[k][0] = upper ? a4.z : o4.x; r[k][1] = upper ? o4.x : o4.y; r[k][2] = upper ? o4.y : o4.z;
                    r[k][3] = upper ? o4.z : a4.x; r[k][4] = a4.y;
                } else {
                    const float4 d4 = __ldg(g.dc + q);
                    r[k][0] = o4.x; r[k][1] = o4.y; r[k][2] = o4.z; r[k][3] = a4.x; r[k][4] = a4.y; r[k][5] = a4.z;
                    r[k][6] = d4.x; r[k][7] = d4.y; r[k][8] = d4.z;
                }
                solid[k] = upper ? 0.0f : o4.w;
            }
            bool odd = false;
#pragma unroll
            for (int k = 0; k < NC; ++k)
#pragma unroll
                for (int m = 0; m < NP; ++m) val[k][m] = mqp::widen_normal(r[k][m], odd);
            if (odd)   // subnormals, infinities, NaN
#pragma unroll
                for (int k = 0; k < NC; ++k)
#pragma unroll
                    for (int m = 0; m < NP; ++m) val[k][m] = (double)r[k][m];
            c0 = solid[0] > 0.5f;
            c1 = solid[1] > 0.5f;
        }
        const unsigned m0 = __ballot_sync(FULL, c0), m1 = NC == 2 ? __ballot_sync(FULL, c1) : 0u;
        if (move) mask = NC == 2 ? (((m0 >> base) & 15u) | (((m1 >> base) & 15u) << 4)) : ((m0 >> base) & 255u);
        return t;
    };
    auto put_fractions = [&](double t) {
        if (b.nearest) t = 0.0;
        const double omt = 1.0 - t;
        if (gl < 3) { tw[2 * gl] = omt; tw[2 * gl + 1] = t; }
    };

    for (uint32_t iter = 1;; ++iter) {
        if (turn) {
            // ---- groups without an ion take the next one of the queue
            bool got = false;
            for (;;) {
                const unsigned need = __ballot_sync(FULL, !have && !drained && gl == 0);
                if (!need) break;
                uint32_t slot = first;
                const unsigned later = __ballot_sync(FULL, !have && !drained && gl == 0 && !fresh);
                if (later) {
                    uint32_t q = 0;
                    const int leader = __ffs(later) - 1;
                    if (lane == leader) q = atomicAdd(head, (uint32_t)__popc(later));
                    q = __shfl_sync(FULL, q, leader) + groups;
                    if (!fresh) slot = q + __popc(later & ((1u << base) - 1u));
                }
                if (!have && !drained) {
                    fresh = false;
                    if (slot >= count) drained = true;
                    else {
                        uint32_t done = 0;
                        id = slot;
                        if (from_hand) { const uint2 e = hand[slot]; id = (uint32_t)MQ_CHK(e.x, n, MQ_SITE_F64_ION); done = e.y; }
                        if (io.status[id] == 0) {
                            have = got = true;
                            jid = io.jid[id];
                            const JobC& jc = jobs[jid];
                            x = d == 0 ? io.x[id] : d == 1 ? io.y[id] : io.z[id];
                            v = d == 0 ? io.vx[id] : d == 1 ? io.vy[id] : io.vz[id];
                            rng = io.rng[id]; age = io.steps[id]; ncoll = io.ncoll[id]; leg = io.leg[id];
                            // steps to the time-out (one at least) or to the end of this call's share
                            left = age < b.max_steps ? b.max_steps - age : 1u;
                            left = min(left, max_more - done);
                            steps_total += gl == 0 ? left : 0u;   // corrected when the ion ends before that
                            use_ac = jc.use_ac != 0;
                            w_tone = is_ac ? jc.w_ac : b.w_rf;
                            const double amp = is_ac ? jc.v_ac : b.v_rf;
                            kick = G == 16 && drives ? amp : jc.qmdt;
                            const float nsd_up = jc.nsd == 0.0 ? 0.0f : mag_up(jc.nsd);
                            nsd2 = __fmul_ru(__fmul_ru(nsd_up, nsd_up), 1.00001f);
                            ub0 = __fmul_ru(__fmul_ru(nsd_up, mag_up(6.0 * jc.s_gas)), 1.00001f);
                            double s0, c0;
                            mqp::sincos2pi(is_ac ? io.ph_ac[id] : io.ph_rf[id], &s0, &c0);
                            ph = second ? s0 : c0;
                            tab = is_ac ? ac_tab + (size_t)jc.tab * tlen : rf_tab;
                            ci = -1;
                            if (G == 16) {     // the amplitudes of the first step
                                double s1, c1;
                                table_get(tab, tlen, w_tone, age, &s1, &c1);
                                if (drives) xch[13 + (is_ac ? 1 : 0)] = amp * (s1 * c0 + c1 * s0);
                            } else {
                                coef = amp;
                            }
                        } else if (gl == 0 && hands) atomicSub(&ctr->open, 1u);
                    }
                }
            }
            if (!__any_sync(FULL, have)) break;
            if (__any_sync(FULL, got)) {
                put_fractions(refill(have && ci < 0, mqp::div_rn(x, h, inv_h)));
                if (G == 4 && got) table_get(tab, tlen, w_tone, age, &S, &Cc);
                __syncwarp();
            }
            turn = false;
        }

        // ---- one step. A group without an ion computes on stale values and keeps nothing.
        // asked for here: the drive's sine and cosine of the next step
        double S1 = 0.0, C1 = 0.0;
        if (have && drives) table_get(tab, tlen, w_tone, age + 1, &S1, &C1);
        const uint64_t r1 = xs_step(rng);   // the first draw of this step's collision, if there is one
        double dr;
        if (G == 16) {
            dr = xch[13 + (chain / 3 == 1 ? 1 : 0)];
            if (chain / 3 == 1 && !use_ac) dr = 0.0;
        } else {
            dr = (second ? Cc : S) * ph;
            dr = dr + shfl_d(dr, lane ^ 2);
            dr = coef * dr;
        }
        // ---- trilinear weights of the lane's corners and their products
        {
            const double wy = tw[2 + ((cn >> 1) & 1)], wz = tw[4 + (cn & 1)];
#pragma unroll
            for (int k = 0; k < NC; ++k) {
                const double w = tw[G == 16 ? cn >> 2 : k] * wy * wz;
#pragma unroll
                for (int m = 0; m < NP; ++m)
                    if (G == 4 || m < 4) prod[((upper ? 5 : 0) + m) * kRow + cn + 4 * k] = w * val[k][m];
                    else if (!upper) prod[m * kRow + cn] = w * val[k][m];
            }
        }
        __syncwarp();
        // ---- sums over the corners in order, one per lane (G = 16) or one per field (G = 4)
        double acc[NS];
#pragma unroll
        for (int f = 0; f < NS; ++f) {
            const double2* row = reinterpret_cast<const double2*>(prod + (chain + 3 * f) * kRow);
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const double2 p = row[c];
                acc[f] = c == 0 ? plus_zero(p.x) : acc[f] + p.x;
                acc[f] = acc[f] + p.y;
            }
        }
        if (G == 16) {
            // sums times amplitudes | drive products of the next step
            const double m = (drives ? (second ? C1 : S1) : dr) * (drives ? ph : acc[0]);
            if (gl < 13) xch[gl] = gl >= 6 && gl < 9 ? acc[0] : m;
            __syncwarp();
            const double e2 = xch[i0] + xch[i1];       // RF + AC | sin cos0 + cos sin0
            const double e = e2 + xch[6 + d];
            const double k = kick * (drives ? e2 : e);  // velocity change | amplitude
            if (gl == 9 || gl == 11) xch[gl == 9 ? 13 : 14] = k;
            v += k;
        } else {
            const double srf = shfl_d(dr, base);
            double sac = shfl_d(dr, base + 1);
            if (!use_ac) sac = 0.0;
            v += kick * (srf * acc[0] + sac * acc[NS / 2] + acc[NS - 1]);
            S = S1;
            Cc = C1;
        }
        x += v * dt;
        age += 1;
        left -= 1;
        // What the end of the step may have to deal with, found while the FP64 pipe works on the new
        // position: a collision, another cell, a limit. Most steps have none and skip it all.
        const double gx = mqp::div_rn(x, h, inv_h);
        double t = gx - cell;
        bool maybe;
        if (!b.legacy_coll) {
            // candidate only if u < nsd (|v| + 6 s), that is u - 6 nsd s < nsd |v|: first in FP32, the
            // left side from below, the right from above and squared
            const float vf = mag_up(v), sq = __fmul_ru(vf, vf);
            const float s2 = __fadd_ru(__shfl_sync(FULL, sq, base), __fadd_ru(__shfl_sync(FULL, sq, base + 1), __shfl_sync(FULL, sq, base + 2)));
            const float du = __fadd_rd((float)(uint32_t)(r1 >> 40) * 0x1.0p-24f, -ub0);
            rng = r1;   // one draw every step
            maybe = have && !(du >= 0.0f && __fmul_rd(du, du) >= __fmul_ru(nsd2, s2));
        } else {
            leg -= 1;
            maybe = have && leg <= 0;
        }
        const bool moved = have && gl < 3 && (unsigned)__double2hiint(t) >= 0x3ff00000u;
        const bool edge = have && ((unsigned)(__double2hiint(x) - in_lo) >= in_n || mask != 0u || left == 0u);
        bool put = false, give = false;
        int32_t status = 0;
        const bool some = __any_sync(FULL, maybe || moved || edge);
        // ---- collisions
        if (some && __any_sync(FULL, maybe)) {
            const JobC& jc = jobs[have ? jid : 0u];
            const double v0 = shfl_d(v, base), v1 = shfl_d(v, base + 1), v2 = shfl_d(v, base + 2);
            const double vm = sqrt(v0 * v0 + v1 * v1 + v2 * v2);
            if (!b.legacy_coll) {
                const double bound = vm + 6.0 * jc.s_gas;
                const bool cand = maybe && xs_unit(r1) < jc.nsd * bound;
                if (__any_sync(FULL, cand)) {
                    uint64_t r = r1, ra = 0, rb = 0;   // six draws: two per axis, in axis order
#pragma unroll
                    for (int k = 0; k < 3; ++k) {
                        r = xs_step(r);
                        if (k == d) ra = r;
                        r = xs_step(r);
                        if (k == d) rb = r;
                    }
                    const double vg = jc.s_gas * mqp::gauss(xs_unit(ra), xs_unit(rb));
                    const double gv = v - vg;
                    const double g0 = shfl_d(gv, base), g1 = shfl_d(gv, base + 1), g2 = shfl_d(gv, base + 2);
                    const double gm = sqrt(g0 * g0 + g1 * g1 + g2 * g2);
                    r = xs_step(r);
                    const bool hit = cand && xs_unit(r) * bound < gm;
                    if (cand) rng = r;
                    if (__any_sync(FULL, hit)) {
                        r = xs_step(r);
                        const double c = 2.0 * xs_unit(r) - 1.0;
                        r = xs_step(r);
                        double sp, cp;
                        mqp::sincos2pi(xs_unit(r), &sp, &cp);
                        const double omc = 1.0 - c * c;
                        const double sn = sqrt(omc > 0.0 ? omc : 0.0);
                        const double nn = d == 2 ? c : sn * (d == 0 ? cp : sp);
                        const double vn = v - jc.mr * gv + jc.mr * gm * nn;
                        if (hit) { v = vn; rng = r; ncoll += 1; }
                    }
                }
            } else {
                uint64_t r = r1;
                const bool hit = maybe && vm > jc.floor_v;
                if (__any_sync(FULL, hit)) {
                    const uint64_t r2 = xs_step(r1), r3 = xs_step(r2);
                    const double c = 2.0 * xs_unit(r1) - 1.0;
                    double sp, cp;
                    mqp::sincos2pi(xs_unit(r2), &sp, &cp);
                    const double omc = 1.0 - c * c;
                    const double sn = sqrt(omc > 0.0 ? omc : 0.0);
                    const double dd = d == 2 ? c : sn * (d == 0 ? cp : sp);
                    const double k1 = 1.0 - jc.mr, k2 = jc.mr * vm;
                    const double vn = v * k1 + k2 * dd;
                    if (hit) { v = vn; r = r3; ncoll += 1; }
                }
                const double u = xs_unit(r);
                const double mfp = -mqp::log_(u > 1e-7 ? u : 1e-7) * jc.mfp_mean;
                const double n0 = shfl_d(v, base), n1 = shfl_d(v, base + 1), n2 = shfl_d(v, base + 2);
                const double vn = sqrt(n0 * n0 + n1 * n1 + n2 * n2);
                double st = floor(mfp / (vn > 1e-3 ? vn : 1e-3) / dt);
                if (st < 1.0) st = 1.0;
                if (maybe) { rng = r; leg = !(st < 2147483647.0) ? 2147483647 : (int32_t)st; }
            }
        }
        if (some && __any_sync(FULL, moved)) t = refill(have, gx);
        put_fractions(t);
        // ---- termination tests: exit, return, box, conductor, time-out
        if (some && __any_sync(FULL, edge || (have && mask != 0u))) {
            const unsigned th = (unsigned)__double2hiint(t);
            const long long bx = __double_as_longlong(x);
            const long long kx = order_key(bx);
            const bool in = !is_nan_bits(bx) && kx > order_key(__double_as_longlong(b.crash_z0)) &&
                            kx < order_key(__double_as_longlong(b.crash_z1));
            const unsigned own = (gt_pos(bx, __double_as_longlong(b.z_exit)) ? 1u : 0u) |
                                 (lt_pos(bx, __double_as_longlong(b.z_return)) ? 2u : 0u) | (in ? 4u : 0u);
            const unsigned zf = __shfl_sync(FULL, own, base + 2);
            const unsigned out = (__ballot_sync(FULL, lt_zero(bx) || gt_pos(bx, __double_as_longlong(b.lim[d]))) >> base) & 7u;
            const unsigned hb = (__ballot_sync(FULL, th >= 0x3fe00000u && th < 0x7ff00000u) >> base) & 7u;   // t >= 0.5
            const unsigned near = ((hb & 1u) << 2) | (hb & 2u) | ((hb >> 2) & 1u);                             // nearest node's corner
            if (have) {
                status = (zf & 1u) ? 3 : (zf & 2u) ? 2 : out ? 4 : 0;
                if (status == 0 && (zf & 4u) && ((mask >> near) & 1u)) status = 1;
                if (status == 0 && age >= b.max_steps) status = 5;
                put = status != 0 || left == 0u;
            }
        }
        if (hands && iter % kPollSteps == 0) {   // few ions left: they go on in wider groups
            const uint32_t open = *(volatile uint32_t*)&ctr->open, taken = *(volatile uint32_t*)head;
            if (__shfl_sync(FULL, (open <= hand_at && (uint64_t)taken + groups >= count) ? 1 : 0, 0) != 0) {
                give = have && !put;
                drained = true;
                turn = true;
            }
        }
        __syncwarp();
        if (__any_sync(FULL, put || give)) {
            turn = true;
            if (put || give) {
                if (gl < 3) {
                    (gl == 0 ? io.x : gl == 1 ? io.y : io.z)[id] = x;
                    (gl == 0 ? io.vx : gl == 1 ? io.vy : io.vz)[id] = v;
                }
                if (gl == 0) {
                    io.rng[id] = rng; io.steps[id] = age; io.ncoll[id] = ncoll; io.leg[id] = leg; io.status[id] = status;
                    steps_total -= left;
                    if (give) hand[MQ_CHK(atomicAdd(&ctr->handed, 1u), hand_at, MQ_SITE_F64_HAND)] = make_uint2(id, max_more - left);
                    else {
                        if (hands) atomicSub(&ctr->open, 1u);
                        live += status == 0 ? 1u : 0u;
                    }
                }
                have = false;
            }
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        steps_total += __shfl_down_sync(FULL, steps_total, o);
        live += __shfl_down_sync(FULL, live, o);
    }
    if (lane == 0) {
        if (steps_total) atomicAdd(&ctr->steps, steps_total);
        if (live) atomicAdd(&ctr->live, live);
    }
}

// ---------------------------------------------------------------- one lane per ion
// For long lists with collisions on most steps, legacy ones or those of a dense gas: with eight ions to a warp some ion
// has one on nearly every step and the warp pays its hundred FP64 operations for that ion alone, with 32 ions it pays them
// once for all that have one. Bound by the FP64 pipe like the groups: with legacy collisions 15.7 us a step for up to 128
// ions per SM, 13.8 for each further 128 (0.1 mm channel), whether they live or not, where the groups take 1.1 to 1.4 us for
// each thousand live ones; with a thermal gas of 5 Pa 25 us, and 1.8 (launch_f64_step has the rules). Every operation is that
// of the groups, in its order. One kernel of this form stepped all FP64 ions before the groups came.
// f32 -> f64 as mqp::widen_normal, other values included: as a branch, since a selected conversion is paid on every value
// (26,000 ions, 2,000 steps 66.6 -> 57.2 ms)
__device__ __forceinline__ double widen(float f) {
    const uint32_t u = __float_as_uint(f);
    const uint32_t e = (u >> 23) & 0xFFu;
    if (e - 1u >= 0xFEu && (u & 0x7FFFFFFFu) != 0u) return (double)f;
    const uint32_t sign = u & 0x80000000u;
    const uint32_t hi = (u & 0x7FFFFFFFu) ? (sign | ((e + 896u) << 20) | ((u & 0x7FFFFFu) >> 3)) : sign;
    return __hiloint2double((int)hi, (int)(u << 29));
}

template <bool LEGACY>
__global__ void __launch_bounds__(128)
k_f64_lane(DevGrid g, Batch b, const JobC* __restrict__ jobs, const double2* __restrict__ rf_tab, const double2* __restrict__ ac_tab,
           uint32_t tlen, DevIons io, uint32_t n, uint32_t max_more, F64Ctrs* __restrict__ ctr) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    uint32_t done = 0;
    int32_t status = 1;
    if (i < n && io.status[i] == 0) {
        const JobC jc = jobs[io.jid[i]];
        const double2* tac = ac_tab + (size_t)jc.tab * tlen;
        double x[3] = {io.x[i], io.y[i], io.z[i]};
        double v[3] = {io.vx[i], io.vy[i], io.vz[i]};
        uint64_t rng = io.rng[i];
        uint32_t age = io.steps[i], ncoll = io.ncoll[i];
        int32_t leg = io.leg[i];
        status = 0;
        double rs, rc, as_, ac;
        mqp::sincos2pi(io.ph_rf[i], &rs, &rc);
        mqp::sincos2pi(io.ph_ac[i], &as_, &ac);
        const double dt = b.dt, qmdt = jc.qmdt, h = g.h;
        const int32_t nn[3] = {g.nx, g.ny, g.nz};
        const long long top[3] = {__double_as_longlong((double)(g.nx - 2)), __double_as_longlong((double)(g.ny - 2)),
                                  __double_as_longlong((double)(g.nz - 2))};
        const size_t nx = (size_t)g.nx, ny = (size_t)g.ny;
        // the cell of the position and its fractions
        double t[3];
        int32_t c[3];
        auto locate = [&]() {
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                const double gx = mqp::div_rn(x[d], h, g.inv_h);
                c[d] = cell_lo_bits(gx, nn[d], top[d]);
                t[d] = gx - i2d_bits(c[d]);
            }
        };
        auto node = [&](int32_t ci, int32_t cj, int32_t ck) {
            const size_t q = (size_t)ci + nx * ((size_t)cj + ny * (size_t)ck);
            return (size_t)MQ_CHK(q, nx * ny * (size_t)g.nz, MQ_SITE_F64_FIELD);
        };
        locate();
        while (done < max_more) {
            double S, Cc, Sa = 0.0, Ca = 0.0;
            table_get(rf_tab, tlen, b.w_rf, age, &S, &Cc);
            const double srf = b.v_rf * (S * rc + Cc * rs);
            double sac = 0.0;
            if (jc.use_ac) {
                table_get(tac, tlen, jc.w_ac, age, &Sa, &Ca);
                sac = jc.v_ac * (Sa * ac + Ca * as_);
            }
            // fields_at: one pass over the 8 corners, weights (1-t, t) in order i, j, k
            if (b.nearest) t[0] = t[1] = t[2] = 0.0;
            double er[3] = {0.0, 0.0, 0.0}, ea[3] = {0.0, 0.0, 0.0}, ed[3] = {0.0, 0.0, 0.0};
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const int di = k >> 2, dj = (k >> 1) & 1, dk = k & 1;
                const double w = (di ? t[0] : 1.0 - t[0]) * (dj ? t[1] : 1.0 - t[1]) * (dk ? t[2] : 1.0 - t[2]);
                const size_t q = node(c[0] + di, c[1] + dj, c[2] + dk);
                const float4 r = __ldg(g.rf + q), a = __ldg(g.ac + q), o = __ldg(g.dc + q);
                er[0] += w * widen(r.x); er[1] += w * widen(r.y); er[2] += w * widen(r.z);
                ea[0] += w * widen(a.x); ea[1] += w * widen(a.y); ea[2] += w * widen(a.z);
                ed[0] += w * widen(o.x); ed[1] += w * widen(o.y); ed[2] += w * widen(o.z);
            }
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                v[d] += qmdt * (srf * er[d] + sac * ea[d] + ed[d]);
                x[d] += v[d] * dt;
            }
            age += 1;
            done += 1;
            if (LEGACY && --leg <= 0) {
                const double vm = sqrt(v[0] * v[0] + v[1] * v[1] + v[2] * v[2]);
                if (vm > jc.floor_v) {
                    const double cth = 2.0 * mqp::xs_next(&rng) - 1.0;
                    double sp, cp;
                    mqp::sincos2pi(mqp::xs_next(&rng), &sp, &cp);
                    const double omc = 1.0 - cth * cth;
                    const double sn = sqrt(omc > 0.0 ? omc : 0.0);
                    const double dd[3] = {sn * cp, sn * sp, cth};
                    const double k1 = 1.0 - jc.mr, k2 = jc.mr * vm;
#pragma unroll
                    for (int d = 0; d < 3; ++d) v[d] = v[d] * k1 + k2 * dd[d];
                    ncoll += 1;
                }
                const double u = mqp::xs_next(&rng);
                const double mfp = -mqp::log_(u > 1e-7 ? u : 1e-7) * jc.mfp_mean;
                const double vn = sqrt(v[0] * v[0] + v[1] * v[1] + v[2] * v[2]);
                double st = floor(mfp / (vn > 1e-3 ? vn : 1e-3) / dt);
                if (st < 1.0) st = 1.0;
                leg = !(st < 2147483647.0) ? 2147483647 : (int32_t)st;
            }
            if (!LEGACY) {
                const double vm = sqrt(v[0] * v[0] + v[1] * v[1] + v[2] * v[2]);
                const double bound = vm + 6.0 * jc.s_gas;
                if (mqp::xs_next(&rng) < jc.nsd * bound) {
                    double gv[3];
#pragma unroll
                    for (int d = 0; d < 3; ++d) {
                        const double u1 = mqp::xs_next(&rng), u2 = mqp::xs_next(&rng);
                        const double vg = jc.s_gas * mqp::gauss(u1, u2);
                        gv[d] = v[d] - vg;
                    }
                    const double gm = sqrt(gv[0] * gv[0] + gv[1] * gv[1] + gv[2] * gv[2]);
                    if (mqp::xs_next(&rng) * bound < gm) {
                        const double cth = 2.0 * mqp::xs_next(&rng) - 1.0;
                        double sp, cp;
                        mqp::sincos2pi(mqp::xs_next(&rng), &sp, &cp);
                        const double omc = 1.0 - cth * cth;
                        const double sn = sqrt(omc > 0.0 ? omc : 0.0);
                        const double dd[3] = {sn * cp, sn * sp, cth};
#pragma unroll
                        for (int d = 0; d < 3; ++d) v[d] = v[d] - jc.mr * gv[d] + jc.mr * gm * dd[d];
                        ncoll += 1;
                    }
                }
            }
            const long long bx = __double_as_longlong(x[0]), by = __double_as_longlong(x[1]), bz = __double_as_longlong(x[2]);
            if (gt_pos(bz, __double_as_longlong(b.z_exit))) status = 3;
            else if (lt_pos(bz, __double_as_longlong(b.z_return))) status = 2;
            else if (lt_zero(bx) || lt_zero(by) || lt_zero(bz) || gt_pos(bx, __double_as_longlong(b.lim[0])) ||
                     gt_pos(by, __double_as_longlong(b.lim[1])) || gt_pos(bz, __double_as_longlong(b.lim[2])))
                status = 4;
            else {
                locate();
                if (x[2] > b.crash_z0 && x[2] < b.crash_z1) {   // the nearest node is a conductor
                    const size_t q = node(c[0] + (t[0] >= 0.5), c[1] + (t[1] >= 0.5), c[2] + (t[2] >= 0.5));
                    if (__ldg(&g.rf[q].w) > 0.5f) status = 1;
                }
                if (status == 0 && age >= b.max_steps) status = 5;
            }
            if (status != 0) break;
        }
        io.x[i] = x[0]; io.y[i] = x[1]; io.z[i] = x[2];
        io.vx[i] = v[0]; io.vy[i] = v[1]; io.vz[i] = v[2];
        io.rng[i] = rng; io.steps[i] = age; io.ncoll[i] = ncoll; io.leg[i] = leg; io.status[i] = status;
    }
    unsigned long long s = done;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(FULL, s, o);
    const uint32_t live = __popc(__ballot_sync(FULL, status == 0));
    if ((threadIdx.x & 31) == 0) {
        if (s) atomicAdd(&ctr->steps, s);
        if (live) atomicAdd(&ctr->live, live);
    }
}

// counters of one round of launches: n open ions, nothing taken or handed on
__global__ void k_f64_begin(F64Ctrs* ctr, uint32_t n) {
    ctr->live = ctr->head_a = ctr->head_b = ctr->handed = 0;
    ctr->open = n;
}

__global__ void k_dc_combine(const float4* b0, const float4* b1, const float4* b2, const float4* b3,
                             float v0, float v1, float v2, float v3, float4* out, size_t n) {
    size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= n) return;
    // e[d] += (v[b] as f32) * dc[b][n][d], bases in order (channel.rs:223); explicit
    // round-to-nearest multiply and add keep it a two-rounding sequence like the host.
    float ex = 0.0f, ey = 0.0f, ez = 0.0f;
    const float4* B[4] = {b0, b1, b2, b3};
    const float V[4] = {v0, v1, v2, v3};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        if (!B[k]) continue;
        float4 e = B[k][q];
        ex = __fadd_rn(ex, __fmul_rn(V[k], e.x));
        ey = __fadd_rn(ey, __fmul_rn(V[k], e.y));
        ez = __fadd_rn(ez, __fmul_rn(V[k], e.z));
    }
    out[q] = make_float4(ex, ey, ez, 0.0f);
}

__global__ void k_summarize(DevIons io, uint32_t n, uint32_t njobs, unsigned long long* cnt) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    uint32_t j = io.jid[i];
    if (j >= njobs) return;
    int32_t st = io.status[i];
    int slot = st == 1 ? 0 : st == 2 ? 1 : st == 3 ? 2 : st == 4 ? 3 : 4;
    unsigned long long* c = cnt + (size_t)j * kCounters;
    atomicAdd(c + slot, 1ull);
    atomicAdd(c + 5, 1ull);
    atomicAdd(c + 6, (unsigned long long)io.ncoll[i]);
    atomicAdd(c + 7, (unsigned long long)io.steps[i]);
}

inline unsigned blocks_for(size_t n, unsigned t) { return (unsigned)((n + t - 1) / t); }

}  // namespace

cudaError_t launch_inject(const mqp::Batch& b, JobTable jt, DevIons io, uint32_t n, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    k_inject<<<blocks_for(n, 128), 128, 0, s>>>(b, jt, io, n);
    return cudaGetLastError();
}

cudaError_t launch_f64_step(DevGrid g, const mqp::Batch& b, const mqp::JobC* jc, const double2* rf_tab,
                            const double2* ac_tab, uint32_t tlen, DevIons io, uint32_t n, uint32_t live, double cand,
                            uint32_t* steps, F64Ctrs* ctr, uint2* hand, cudaStream_t s, uint32_t* kernels) {
    if (n == 0) return cudaSuccess;
    int dev = 0, sms = 0;
    cudaError_t e;
    if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
    if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
    // one block per SM: the shared memory asked for lets no second one in
    if ((e = cudaFuncSetAttribute(k_f64_step<4>, cudaFuncAttributeMaxDynamicSharedMemorySize, kPad)) != cudaSuccess) return e;
    if ((e = cudaFuncSetAttribute(k_f64_step<16>, cudaFuncAttributeMaxDynamicSharedMemorySize, kPad)) != cudaSuccess) return e;
    k_f64_begin<<<1, 1, 0, s>>>(ctr, n);
    const uint32_t wide = f64_hand_entries(sms);
    // One ion to a lane while more live than so many per SM for each 128 per SM in the list, looked at again after a round.
    // Legacy collisions, 2,000 steps, groups alone / so: 10,000 ions 29 / 29 ms, 15,000 45 / 33, 26,000 76 / 57, 40,000 109 / 85; 200
    // steps of 200,000 ions 44 / 30; 40,000 ions to their end (20,000 steps) 745 / 702. Thermal collisions: where a resting ion
    // is a candidate on 14 in 100 steps or more (1.7 Pa for the ions and step of a mass scan; below, the groups are faster), 200,000
    // ions, 200 steps at 2 Pa 58 / 53 ms, 5 Pa 73 / 53, 30 Pa 80 / 53.
    const uint64_t waves = ((uint64_t)n + 128u * (uint32_t)sms - 1u) / (128u * (uint32_t)sms);
    const uint64_t line = (b.legacy_coll ? 72u : 78u + (uint32_t)(5.0 / std::fmax(cand, 0.14))) * (uint32_t)sms * waves;
    uint32_t max_more = *steps;
    if ((b.legacy_coll || cand >= 0.14) && live > line) {
        const uint32_t round = b.legacy_coll ? kLaneRound : kLaneRound / 8;
        *steps = max_more = max_more < round ? max_more : round;
        const unsigned blocks = blocks_for(n, 128);
        if (b.legacy_coll) k_f64_lane<true><<<blocks, 128, 0, s>>>(g, b, jc, rf_tab, ac_tab, tlen, io, n, max_more, ctr);
        else k_f64_lane<false><<<blocks, 128, 0, s>>>(g, b, jc, rf_tab, ac_tab, tlen, io, n, max_more, ctr);
        *kernels += 2;
    } else if (n <= wide) {
        k_f64_step<16><<<sms, kBlock, kPad, s>>>(g, b, jc, rf_tab, ac_tab, tlen, io, n, max_more, ctr, nullptr, 0, 0);
        *kernels += 2;
    } else {
        k_f64_step<4><<<sms, kBlock, kPad, s>>>(g, b, jc, rf_tab, ac_tab, tlen, io, n, max_more, ctr, hand, hand ? wide : 0, 0);
        *kernels += 2;
        if (hand) {
            k_f64_step<16><<<sms, kBlock, kPad, s>>>(g, b, jc, rf_tab, ac_tab, tlen, io, n, max_more, ctr, hand, 0, 1);
            *kernels += 1;
        }
    }
    return cudaGetLastError();
}

cudaError_t launch_phase_table(double w, uint32_t len, double2* out, cudaStream_t s) {
    if (len == 0) return cudaSuccess;
    k_phase_table<<<blocks_for(len, 256), 256, 0, s>>>(w, len, out);
    return cudaGetLastError();
}

cudaError_t launch_dc_combine(const float4* b0, const float4* b1, const float4* b2, const float4* b3,
                              float v0, float v1, float v2, float v3, float4* out, size_t n, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    k_dc_combine<<<blocks_for(n, 256), 256, 0, s>>>(b0, b1, b2, b3, v0, v1, v2, v3, out, n);
    return cudaGetLastError();
}

cudaError_t launch_summarize(DevIons io, uint32_t n, uint32_t njobs, unsigned long long* counters, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    k_summarize<<<blocks_for(n, 256), 256, 0, s>>>(io, n, njobs, counters);
    return cudaGetLastError();
}

}  // namespace mqd

MQ_CHECK_READER(mq_check_read_f64)
