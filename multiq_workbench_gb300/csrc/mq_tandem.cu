// Nine-channel tandem transport on the GPU: a group of lanes per track, every track on
// the global clock, FP64 state, compiled without FMA contraction so that every track's
// arithmetic equals the CPU restatement of trapsim::Model::advance bit for bit.
//
// Reference: simulation/trapsim/src/lib.rs:69-103 (cube_field, transport_step),
// lib.rs:176-276 (Model::advance: region fields, routing), lib.rs:338-385 (enter / leave),
// simulation/mqviz/src/world.rs:265-314 (fields_at, gate_delta, is_crash), world.rs:471-488
// (collide).
#include <cmath>
#include <cstring>
#include <string>
#include <utility>
#include <vector>

#include "mq_cube_geom.h"
#include "mq_phys.h"
#include "mq_tandem.h"
#include "mq_tandem_internal.h"
#include "mq_check.h"
#include "mq_f64dev.h"

namespace {

constexpr double Z_EXIT = 18.6e-3;     // world.rs:21
constexpr double Z_RETURN = 0.5e-3;    // world.rs:22
constexpr int R_SPLIT = 0, R_COMBINE = 10, R_LOST = 11, R_BACK = 12, R_DETECTED = 13;
constexpr int kNC = 21;                 // counters per port (mq_port_counts)
constexpr size_t kCntBytes = (9 * kNC * 4 + 7) / 8 * 8;               // port counters, then six 8-byte step counters
constexpr size_t kTail = kCntBytes + 6 * sizeof(unsigned long long);
constexpr size_t kStageMax = 256 * 1024;

using namespace mqf;

struct TSpec { double qmdt, s_ion, mr, nsd; };

struct TPort {                  // one port's channel grid and drive
    int32_t kn[3], idle;
    double kh, inv_kh, lim[3];   // spacing [m], its correctly rounded reciprocal, box limits
    const float4 *rf, *ac, *dc, *gate;
};

// Cube geometry in FP32 (mm, growth 0), for the filter that settles all but the points near a surface
struct CubeF {
    float size, c0, pitch, half_d, t_pcb, gap, ptd, stem_r, clear_r, rod_hole, l_ext, cap_reach, cap_r, ap_r;
    float ent_b, ent_c;      // entrance axis: along z, along x
    float near;              // distances [mm] closer than this are left to the exact test,
    float round_port, round_post;   // and fractions beyond these
    int32_t n, array, ent_axis, ent_side, ent_cell0, ent_cell1, ext_axis, ext_side, ext_cell0, ext_cell1;
};

struct TConst {
    mq_cube_geom cube;
    int32_t cn[3];
    double clo[3], ch_mm, inv_ch_mm;
    const float4* crf;
    const float4* cdc[2];
    TPort port[9];
    double axis, seam, size, ap_r, l_ext_m, dt, s_gas, gate_v;
    double mouth[9][2];
    double ent_b, ent_c;   // entrance axis centre (mm): along z, along x
    TSpec sp[8];
    CubeF F;
    // high words of the positions (m) that are out of reach of every cube face and short of the seam
    int32_t in_lo;
    uint32_t in_n[3];
};

struct Tracks {
    double *x, *y, *z, *vx, *vy, *vz;
    uint64_t* rng;
    int32_t *sp, *region, *last;
};

__device__ __forceinline__ float latf(const CubeF& G, int i) { return G.c0 + G.pitch * (float)i; }
__device__ __forceinline__ float hypf2(float u, float v) { return sqrtf(u * u + v * v); }
// v < t, noting in `unsure` when the two are too close to tell
__device__ __forceinline__ bool below(const CubeF& G, float v, float t, bool& unsure) {
    unsure |= !(fabsf(v - t) >= G.near);   // NaN too
    return v < t;
}
// v.round() clamped to [0, hi]
__device__ __forceinline__ int round_near(float v, int hi, float most, bool& unsure) {
    const float r = rintf(v);
    unsure |= !(fabsf(v - r) <= most);
    return r > 0.0f ? (r < (float)hi ? (int)r : hi) : 0;
}
// mqc::classify (geometry.rs:136-205) for one face (axis a, side) of the point: does the point lie in
// an electrode of it?  u: depth below the face, pb / pc: the coordinates along axes a + 1 and a + 2
__device__ bool face_solid(const CubeF& G, int a, int side, float u, float pb, float pc, bool inside, bool& unsure) {
    int pid = 0, pc0 = 0, pc1 = 0;
    if (G.ent_axis == a && G.ent_side == side) { pid = 3; pc0 = G.ent_cell0; pc1 = G.ent_cell1; }
    else if (G.ext_axis == a && G.ext_side == side) {
        pid = 4;
        pc0 = G.ext_cell0; pc1 = G.ext_cell1;
        if (G.array) {
            const float first = 0.5f * (latf(G, 2) + latf(G, 3));
            pc0 = 2 + 2 * round_near((pb - first) / (2.0f * G.pitch), 2, G.round_port, unsure);
            pc1 = 2 + 2 * round_near((pc - first) / (2.0f * G.pitch), 2, G.round_port, unsure);
        }
    }
    const float axis_d = hypf2(pb - 0.5f * (latf(G, pc0) + latf(G, pc0 + 1)), pc - 0.5f * (latf(G, pc1) + latf(G, pc1 + 1)));
    if (below(G, u, 0.0f, unsure)) {   // outside the wall: port rods and end cap
        if (pid == 0) return false;
        bool hit = false;
        if (below(G, u, -G.cap_reach, unsure)) hit = below(G, axis_d, G.cap_r, unsure);
        if (!below(G, u, -G.l_ext, unsure))
            for (int m = 0; m < 4; ++m)
                hit |= below(G, hypf2(pb - latf(G, pc0 + (m >> 1)), pc - latf(G, pc1 + (m & 1))), G.half_d, unsure);
        return hit;
    }
    if (!inside || !below(G, u, G.ptd, unsure)) return false;
    const int ib = round_near((pb - G.c0) / G.pitch, G.n - 1, G.round_post, unsure);
    const int ic = round_near((pc - G.c0) / G.pitch, G.n - 1, G.round_post, unsure);
    const bool rim_b = ib == 0 || ib == G.n - 1, rim_c = ic == 0 || ic == G.n - 1;
    const bool valid = a == 0 ? !rim_b && !rim_c : a == 1 ? !rim_b : true;   // post_valid, geometry.rs:81-86
    const float dd = hypf2(pb - latf(G, ib), pc - latf(G, ic));
    const bool rod = pid != 0 && valid && (unsigned)(ib - pc0) <= 1u && (unsigned)(ic - pc1) <= 1u;
    const bool aperture = pid != 0 && below(G, axis_d, G.ap_r, unsure);
    const bool in_post = below(G, dd, G.half_d, unsure);
    if (rod && in_post) return true;
    if (below(G, u, G.t_pcb, unsure) && !aperture && !(valid && below(G, dd, rod ? G.rod_hole : G.clear_r, unsure))) return true;
    if (valid && !rod) {
        if (below(G, u, G.t_pcb + G.gap, unsure)) return below(G, dd, G.stem_r, unsure);
        return in_post;
    }
    return false;
}

// Executed track-steps by region kind (cube, driven port, idle port): one warp-reduced atomic per warp.
__device__ __forceinline__ void add_steps(unsigned long long* st, uint32_t c, uint32_t p, uint32_t q) {
    c = __reduce_add_sync(0xffffffffu, c);
    p = __reduce_add_sync(0xffffffffu, p);
    q = __reduce_add_sync(0xffffffffu, q);
    if ((threadIdx.x & 31) == 0) {
        if (c) atomicAdd(st + 0, (unsigned long long)c);
        if (p) atomicAdd(st + 1, (unsigned long long)p);
        if (q) atomicAdd(st + 2, (unsigned long long)q);
    }
}

// ---------------------------------------------------------------- the step kernel
// Bound by GB300's FP64 pipe and by latency, as the channel's FP64 kernel (mq_f64.cu), and shaped like it: a
// group of G lanes per track, each lane an axis (position, velocity) and one of the eight cell
// corners (two for G = 4), the sums over the corners side by side in the lanes. With one lane per track
// a step took 32 us. In the cube the electrode test, some hundreds of FP64 operations, is first made in
// FP32, one face of the cube per lane, and exactly only near a surface (CubeF::near); whether a
// track is at a limit at all is read off the high words of its position. Every operation that counts is the
// reference's, in its order: results are bit for bit those of one lane per track.
// G = 16 while the tracks fit one warp per scheduler (two of them in a warp), 4 beyond, where fewer wasted
// lanes count for more; groups take the next track when theirs has made its steps or is lost.
// Measured, whole advance call, 180 tracks and 100 steps, from the mouths 3.45 -> 0.36 ms; kernel, 200,000 tracks and 200
// steps, from the mouths 73 -> 41 ms, through the entrance 50 -> 29.5.
constexpr int kTBlock = 256;
constexpr int kTRow = 10;
constexpr int kTSums = 6 + 12 * kTRow;
constexpr int kTGroup = kTSums + 12;     // doubles of shared memory per group
constexpr int kTPad = 120 * 1024;        // one block per SM

// drive of global steps [s0, s0 + k): rf = V_rf sin(2 pi f_rf t), ac_i = V_ac sin(2 pi f_i t), t = s dt
// (lib.rs:178-182); one thread per step and tone. On the host, a microsecond a step, it took a tenth of
// a large advance. `Out` is float for the mixed engine (no FP64 conversions in its step loop).
struct Tones { double f[10], v[10], dt; };
template <class Out>
__global__ void k_drive(const __grid_constant__ Tones tn, uint64_t s0, uint32_t k, Out* __restrict__ out) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= k * 10u) return;
    const uint32_t q = i / 10u, c = i % 10u;
    const double t = (double)(s0 + q) * tn.dt;
    const double p = tn.f[c] * t;
    double s, co;
    mqp::sincos2pi(p - floor(p), &s, &co);
    out[i] = (Out)(tn.v[c] * s);
}

template <int G>
__global__ void __launch_bounds__(kTBlock, 1)
k_tandem(const __grid_constant__ TConst C, Tracks T, uint32_t n, const double* __restrict__ drive, uint32_t steps,
         uint32_t* __restrict__ counts, unsigned long long* __restrict__ stepc, uint32_t* __restrict__ head) {
    constexpr int GPW = 32 / G;
    constexpr int NC = G == 16 ? 1 : 2;     // corners per lane
    constexpr int NP = G == 16 ? 6 : 12;    // products per corner: RF, AC, DC, gate of three components; G = 16: half of them
    constexpr int NS = G == 16 ? 1 : 4;     // sums per lane
    extern __shared__ __align__(16) double sm[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, gl = lane % G, base = lane - gl;
    const int d = gl % 3;
    double* const tw = sm + (size_t)(threadIdx.x / G) * kTGroup;
    double* const prod = tw + 6;
    double* const xch = tw + kTSums;
    const uint32_t first = (uint32_t)((((warp >> 2) * GPW + lane / G) * 4 + (warp & 3)) * gridDim.x + blockIdx.x);
    const uint32_t groups = gridDim.x * (kTBlock / 32) * GPW;
    // corner index in the order of the sums: 4 di + 2 dj + dk in a port, di + 2 dj + 4 dk in the cube
    const int cn = G == 16 ? gl & 7 : gl;
    const bool upper = G == 16 && gl >= 8;
    const int chain = G == 16 ? (gl < 12 ? gl : gl - 12) : d;   // sum 3 f + d: RF, AC, DC, gate (cube: the first three)

    bool have = false, drained = false, fresh = true, turn = true;
    uint32_t id = 0, k = 0;
    int reg = R_LOST, last = -1, sp = 0;
    uint64_t rng = 1;
    double x = 0.0, v = 0.0, q = 0.0, cell = 0.0, qmdt = 0.0;
    float nsd2 = 0.0f, ub0 = 0.0f;
    bool cube = true, idle = false;
    int32_t ci = -1, cj = -1, ck = -1, nd = 2;
    uint32_t mask = 0, n_cube = 0, n_port = 0, n_idle = 0;
    double gh = 1.0, ginv = 1.0, glim = 0.0;   // grid spacing, its reciprocal, box limit along the axis (port)
    size_t nx = 2, ny = 2;
    const float4 *p_rf = nullptr, *p_ac = nullptr, *p_dc = nullptr, *p_gate = nullptr;
    // the lane's limits in the cube: its size, and the seam (z) or the end of the entrance (y), as keys of their order
    const long long key_size = order_key(__double_as_longlong(C.size));
    const long long key_end = order_key(__double_as_longlong(d == 2 ? C.seam : C.size + C.l_ext_m));
    const double cube_top = (double)(C.cn[d] - 1) - 1e-9;
    double val[NC][NP];
#pragma unroll
    for (int c = 0; c < NC; ++c)
#pragma unroll
        for (int m = 0; m < NP; ++m) val[c][m] = 0.0;

    // constants of the group's region, and the lane's coordinate on its grid: x / h in a port, mm in the cube
    auto enter_region = [&](bool go) {
        if (go) {
            cube = reg == R_SPLIT || reg == R_COMBINE;
            if (cube) {
                nd = C.cn[d]; nx = (size_t)C.cn[0]; ny = (size_t)C.cn[1];
                p_rf = C.crf; p_dc = C.cdc[reg == R_COMBINE ? 1 : 0];
                idle = false;
            } else {
                const TPort& P = C.port[reg - 1];
                nd = P.kn[d]; nx = (size_t)P.kn[0]; ny = (size_t)P.kn[1];
                p_rf = P.rf; p_ac = P.ac; p_dc = P.dc; p_gate = P.gate;
                gh = P.kh; ginv = P.inv_kh; glim = P.lim[d];
                idle = P.idle != 0;
            }
            ci = -1;
        }
    };
    auto coordinate = [&](bool go) {
        if (__any_sync(FULL, go && cube)) { const double qc = x * 1000.0; if (go && cube) q = qc; }
        if (__any_sync(FULL, go && !cube)) { const double qp = mqp::div_rn(x, gh, ginv); if (go && !cube) q = qp; }
    };
    // cell and fractions; corner values of the groups in `go` that changed cell
    auto locate = [&](bool go) -> double {
        double f = q;
        if (__any_sync(FULL, go && cube)) {   // fields.rs:89-96: clamped to the grid, short of its last node
            const double fc = mqp::div_rn(q - C.clo[d], C.ch_mm, C.inv_ch_mm);
            const long long b = __double_as_longlong(fc);
            if (cube) f = lt_zero(b) ? 0.0 : gt_pos(b, __double_as_longlong(cube_top)) ? cube_top : fc;
        }
        double t = f - cell;
        const bool stay = ci >= 0 && (unsigned)__double2hiint(t) < 0x3ff00000u;
        if (__any_sync(FULL, go && gl < 3 && !stay)) {
            const int32_t ca = cell_lo_bits(f, nd, __double_as_longlong(i2d_bits(nd - 2)));
            const double cd = i2d_bits(ca);
            if (go) { cell = cd; t = f - cd; }
            const int32_t ni = __shfl_sync(FULL, ca, base), nj = __shfl_sync(FULL, ca, base + 1), nk = __shfl_sync(FULL, ca, base + 2);
            const bool move = go && (ni != ci || nj != cj || nk != ck);
            bool c0 = false, c1 = false;
            if (move) {
                ci = ni; cj = nj; ck = nk;
                float r[NC][12], solid[2] = {0.0f, 0.0f};
#pragma unroll
                for (int c = 0; c < NC; ++c) {
                    const int m = cn + 4 * c;   // G = 4: corners cn and cn + 4
                    const int lo = m & 1, mid = (m >> 1) & 1, hi = m >> 2;
                    const size_t o = (size_t)(ci + (cube ? lo : hi)) + nx * ((size_t)(cj + mid) + ny * (size_t)(ck + (cube ? hi : lo)));
                    const size_t w = cube ? MQ_CHK(o, (size_t)C.cn[0] * (size_t)C.cn[1] * (size_t)C.cn[2], MQ_SITE_TDM_CUBE)
                                          : MQ_CHK(o, nx * ny * (size_t)C.port[reg - 1].kn[2], MQ_SITE_TDM_PORT);
#pragma unroll
                    for (int z = 0; z < 12; ++z) r[c][z] = 0.0f;
                    // G = 16: lower lanes RF and AC (cube: RF and DC), upper lanes DC and gate
                    if (G == 16) {
                        if (!(cube && upper)) {
                            const float4 u = __ldg((upper ? p_dc : p_rf) + w);
                            r[c][0] = u.x; r[c][1] = u.y; r[c][2] = u.z;
                            solid[c] = upper || cube ? 0.0f : u.w;
                            if (!upper || idle) {
                                const float4 y = __ldg((cube ? p_dc : upper ? p_gate : p_ac) + w);
                                r[c][3] = y.x; r[c][4] = y.y; r[c][5] = y.z;
                            }
                        }
                    } else {
                        const float4 u = __ldg(p_rf + w), y = __ldg((cube ? p_dc : p_ac) + w);
                        r[c][0] = u.x; r[c][1] = u.y; r[c][2] = u.z; r[c][3] = y.x; r[c][4] = y.y; r[c][5] = y.z;
                        solid[c] = cube ? 0.0f : u.w;
                        if (!cube) {
                            const float4 z = __ldg(p_dc + w);
                            r[c][6] = z.x; r[c][7] = z.y; r[c][8] = z.z;
                            if (idle) { const float4 g = __ldg(p_gate + w); r[c][9] = g.x; r[c][10] = g.y; r[c][11] = g.z; }
                        }
                    }
                }
                bool odd = false;
#pragma unroll
                for (int c = 0; c < NC; ++c)
#pragma unroll
                    for (int m = 0; m < NP; ++m) val[c][m] = mqp::widen_normal(r[c][m], odd);
                if (odd)
#pragma unroll
                    for (int c = 0; c < NC; ++c)
#pragma unroll
                        for (int m = 0; m < NP; ++m) val[c][m] = (double)r[c][m];
                c0 = solid[0] > 0.5f;
                c1 = solid[1] > 0.5f;
            }
            const unsigned m0 = __ballot_sync(FULL, c0), m1 = NC == 2 ? __ballot_sync(FULL, c1) : 0u;
            if (move) mask = NC == 2 ? (((m0 >> base) & 15u) | (((m1 >> base) & 15u) << 4)) : ((m0 >> base) & 255u);
        }
        return t;
    };

    for (;;) {
        if (turn) {
            bool got = false;
            for (;;) {   // groups without a track take the next one
                const unsigned need = __ballot_sync(FULL, !have && !drained && gl == 0);
                if (!need) break;
                uint32_t slot = first;
                const unsigned later = __ballot_sync(FULL, !have && !drained && gl == 0 && !fresh);
                if (later) {
                    uint32_t o = 0;
                    const int leader = __ffs(later) - 1;
                    if (lane == leader) o = atomicAdd(head, (uint32_t)__popc(later));
                    o = __shfl_sync(FULL, o, leader) + groups;
                    if (!fresh) slot = o + __popc(later & ((1u << base) - 1u));
                }
                if (!have && !drained) {
                    fresh = false;
                    if (slot >= n) drained = true;
                    else {
                        id = slot;
                        reg = T.region[id];
                        if (reg < R_LOST) {
                            have = got = true;
                            k = 0;
                            x = d == 0 ? T.x[id] : d == 1 ? T.y[id] : T.z[id];
                            v = d == 0 ? T.vx[id] : d == 1 ? T.vy[id] : T.vz[id];
                            rng = T.rng[id]; sp = T.sp[id]; last = T.last[id];
                            qmdt = C.sp[sp].qmdt;
                            const double nsd = C.sp[sp].nsd;
                            const float nsd_up = nsd == 0.0 ? 0.0f : mag_up(nsd);
                            nsd2 = __fmul_ru(__fmul_ru(nsd_up, nsd_up), 1.00001f);
                            ub0 = __fmul_ru(__fmul_ru(nsd_up, mag_up(6.0 * C.s_gas)), 1.00001f);
                        }
                    }
                }
            }
            if (!__any_sync(FULL, have)) break;
            if (__any_sync(FULL, got)) {
                enter_region(got);
                coordinate(got);
                const double t = locate(got);
                if (got && gl < 3) { tw[2 * gl] = 1.0 - t; tw[2 * gl + 1] = t; }
                __syncwarp();
            }
            turn = false;
        }
        // ---- field at the current position (lib.rs:70-88, world.rs:265-302)
        const double* dr = drive + (size_t)(have ? k : 0u) * 10;
        const double rf = dr[0], ac = dr[have && !cube ? reg : 0];
        const uint64_t r1 = xs_step(rng);
        const bool any_cube = __any_sync(FULL, have && cube), any_port = __any_sync(FULL, have && !cube);
        const bool any_idle = __any_sync(FULL, have && idle);
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            const int m = cn + 4 * c, lo = m & 1, mid = (m >> 1) & 1, hi = m >> 2;
            const double wx = tw[cube ? lo : hi], wy = tw[2 + mid], wz = tw[4 + (cube ? hi : lo)];
            const double w = wx * wy * wz;
            double wg = 0.0;
            if (any_idle) wg = C.gate_v * wx * wy * wz;
            if (any_port) {
                if (!cube) {
                    if (G == 16) {
#pragma unroll
                        for (int z = 0; z < 6; ++z) prod[((upper ? 6 : 0) + z) * kTRow + m] = (upper && z >= 3 ? wg : w) * val[c][z % NP];
                    } else {
#pragma unroll
                        for (int z = 0; z < 9; ++z) prod[z * kTRow + m] = w * val[c][z % NP];
                        if (any_idle)
#pragma unroll
                            for (int z = 9; z < 12; ++z) prod[z * kTRow + m] = wg * val[c][z % NP];
                    }
                }
            }
            if (any_cube) {
                if (cube && !upper)
#pragma unroll
                    for (int z = 0; z < 3; ++z) prod[z * kTRow + m] = w * (rf * val[c][z % NP] + val[c][(z + 3) % NP]);
            }
        }
        __syncwarp();
        double acc[NS];
#pragma unroll
        for (int f = 0; f < NS; ++f) {
            acc[f] = 0.0;
            if (f == 0 || (f < 3 && any_port) || any_idle) {
                const double2* row = reinterpret_cast<const double2*>(prod + (chain + 3 * f) * kTRow);
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const double2 p = row[c];
                    acc[f] = c == 0 ? plus_zero(p.x) : acc[f] + p.x;
                    acc[f] = acc[f] + p.y;
                }
            }
        }
        double e;
        if (G == 16) {
            if (any_port) {
                const int f = chain / 3;
                const double m = (f == 0 ? rf : ac) * acc[0];
                if (gl < 12) xch[gl] = cube || f >= 2 ? acc[0] : m;
                __syncwarp();
                e = xch[d] + xch[3 + d] + xch[6 + d];
                e = idle ? e + xch[9 + d] : plus_zero(e);   // + 0.0 where there is no gate
                if (cube) e = xch[d];
            } else {
                e = shfl_d(acc[0], base + d);
            }
        } else {
            e = rf * acc[0] + ac * acc[1 % NS] + acc[2 % NS];
            e = idle ? e + acc[3 % NS] : plus_zero(e);
            if (cube) e = acc[0];
        }
        // ---- transport_step (lib.rs:90-103)
        v += qmdt * e;
        x += v * C.dt;
        if (have) {
            if (cube) ++n_cube;
            else if (idle) ++n_idle;
            else ++n_port;
            k += 1;
        }
        // ---- thermal collisions (world.rs:473-488): first against an FP32 bound, as in mq_f64.cu
        {
            const float vf = mag_up(v), sq = __fmul_ru(vf, vf);
            const float s2 = __fadd_ru(__shfl_sync(FULL, sq, base), __fadd_ru(__shfl_sync(FULL, sq, base + 1), __shfl_sync(FULL, sq, base + 2)));
            const float du = __fadd_rd((float)(uint32_t)(r1 >> 40) * 0x1.0p-24f, -ub0);
            rng = r1;
            const bool maybe = have && !(du >= 0.0f && __fmul_rd(du, du) >= __fmul_ru(nsd2, s2));
            if (__any_sync(FULL, maybe)) {
                const TSpec& S = C.sp[sp];
                const double v0 = shfl_d(v, base), v1 = shfl_d(v, base + 1), v2 = shfl_d(v, base + 2);
                const double vm = sqrt(v0 * v0 + v1 * v1 + v2 * v2);
                const double bound = vm + 6.0 * C.s_gas;
                const bool cand = maybe && xs_unit(r1) < S.nsd * bound;
                if (__any_sync(FULL, cand)) {
                    uint64_t r = r1, ra = 0, rb = 0;
#pragma unroll
                    for (int z = 0; z < 3; ++z) {
                        r = xs_step(r);
                        if (z == d) ra = r;
                        r = xs_step(r);
                        if (z == d) rb = r;
                    }
                    const double vg = C.s_gas * mqp::gauss(xs_unit(ra), xs_unit(rb));
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
                        double sn_, cs_;
                        mqp::sincos2pi(xs_unit(r), &sn_, &cs_);
                        const double omc = 1.0 - c * c;
                        const double sn = sqrt(omc > 0.0 ? omc : 0.0);
                        const double nn = d == 2 ? c : sn * (d == 0 ? cs_ : sn_);
                        const double vn = v - S.mr * gv + S.mr * gm * nn;
                        if (hit) { v = vn; rng = r; }
                    }
                }
            }
        }
        // ---- routing (lib.rs:212-272)
        coordinate(have);
        bool changed = false;   // the track is in another region now
        const int xhi = __double2hiint(x);
        if (any_cube) {
            // inside the posts' reach of no face, before the seam: nothing can happen
            const bool off = have && cube && gl < 3 && (unsigned)(xhi - C.in_lo) >= C.in_n[d];
            if (__any_sync(FULL, off)) {
                // The look at the walls stays off the FP64 pipe: one conversion a lane, limits by the positions' bits, distances
                // in FP32 where these decide. The groups' tracks share the pipe's instructions by eight, not by 32 as single
                // lanes did.
                const float pm = (float)q;
                const float p0 = __shfl_sync(FULL, pm, base), p1 = __shfl_sync(FULL, pm, base + 1), p2 = __shfl_sync(FULL, pm, base + 2);
                bool unsure = false, solid = false;
                {
                    const float l = C.F.size;
                    bool far = false;   // close to a face plane the FP32 `inside` is not to be trusted
                    const bool inside = !below(C.F, p0, 0.0f, far) && !below(C.F, p1, 0.0f, far) && !below(C.F, p2, 0.0f, far) &&
                                        below(C.F, p0, l, far) && below(C.F, p1, l, far) && below(C.F, p2, l, far);
                    unsure = far;
                    for (int f = gl; f < 6; f += G) {
                        const int a = f >> 1, side = f & 1;
                        const float pa = a == 0 ? p0 : a == 1 ? p1 : p2, pb = a == 0 ? p1 : a == 1 ? p2 : p0, pc = a == 0 ? p2 : a == 1 ? p0 : p1;
                        bool un = false;
                        if (face_solid(C.F, a, side, side == 0 ? pa : l - pa, pb, pc, inside, un) && !un) solid = true;
                        unsure |= un;
                    }
                }
                // beyond the cube's size | the seam (z) or the entrance's end (y) | below zero
                const long long bx = __double_as_longlong(x);
                const unsigned own = (gt_key(bx, key_size) ? 1u : 0u) | (gt_key(bx, key_end) ? 2u : 0u) | (lt_zero(bx) ? 4u : 0u);
                const unsigned fx = __shfl_sync(FULL, own, base), fy = __shfl_sync(FULL, own, base + 1), fz = __shfl_sync(FULL, own, base + 2);
                constexpr unsigned GM = G == 32 ? 0xffffffffu : (1u << G) - 1u;
                const bool g_solid = ((__ballot_sync(FULL, solid) >> base) & GM) != 0u, g_unsure = ((__ballot_sync(FULL, unsure) >> base) & GM) != 0u;
                const bool go = have && cube;   // a group that is well inside finds just that
                // off the entrance's axis, where it counts: beyond the cube in y
                bool un = false;
                bool off_axis = !below(C.F, hypf2(p0 - C.F.ent_c, p2 - C.F.ent_b), C.F.ap_r, un);
                const bool beyond = go && (fz & 2u), ask_wall = go && g_unsure, ask_axis = go && (fy & 1u) && un;
                double x0 = 0.0, x1 = 0.0, x2 = 0.0, m0 = 0.0, m1 = 0.0, m2 = 0.0;
                bool blocked = g_solid;
                if (__any_sync(FULL, beyond || ask_wall || ask_axis)) {
                    x0 = shfl_d(x, base); x1 = shfl_d(x, base + 1); x2 = shfl_d(x, base + 2);
                    m0 = shfl_d(q, base); m1 = shfl_d(q, base + 1); m2 = shfl_d(q, base + 2);
                    if (ask_wall) {
                        const double mm[3] = {m0, m1, m2};
                        int sg = 0;
                        blocked = mqc::classify(C.cube, mm, 0.0, &sg) != mqc::ID_FREE;
                    }
                    if (ask_axis) off_axis = mqc::dist2d(m0 - C.ent_c, m2 - C.ent_b) >= C.ap_r;
                }
                if (go) {
                    bool done = false;
                    if (blocked) { reg = R_LOST; done = true; }
                    if (!done && beyond) {
                        const int i = mqc::nearest_port(C.cube, m0, m1);
                        const double* c = C.mouth[i];
                        if (mqc::dist2d(x0 - c[0], x1 - c[1]) < C.ap_r * 0.001) {
                            // enter (lib.rs:338-367)
                            uint32_t* cnt = counts + (size_t)i * kNC;
                            const double depth = x2 - C.seam;
                            if (d < 2) x += C.axis - c[d];
                            if (reg == R_SPLIT) {
                                if (d == 2) x = Z_RETURN + depth;
                                if (gl == 0) {
                                    atomicAdd(cnt + 0, 1u);
                                    if (last >= 0) {
                                        atomicAdd(cnt + 3, 1u);
                                        atomicAdd(cnt + 5 + last, 1u);
                                        if (last != i) atomicAdd(cnt + 4, 1u);
                                    }
                                }
                            } else {
                                if (d == 2) { x = Z_EXIT - depth; v *= -1.0; }
                                if (gl == 0) atomicAdd(cnt + 14, 1u);
                            }
                            reg = 1 + i;
                            changed = done = true;
                        } else if (fz & 1u) { reg = R_LOST; done = true; }
                    }
                    if (!done && (fy & 1u) && off_axis) { reg = R_LOST; done = true; }
                    if (!done) {
                        if (fy & 2u) reg = (reg == R_SPLIT) ? R_BACK : R_DETECTED;
                        else if (((fx | fy | fz) & 4u) || (fx & 1u)) reg = R_LOST;
                    }
                }
            }
        }
        double t = locate(have && !changed && reg < R_LOST);
        if (any_port) {
            // is_crash (world.rs:309-314): outside the box, or the nearest node is a conductor
            const bool port = have && !cube;
            const long long bx = __double_as_longlong(x);
            const unsigned th = (unsigned)__double2hiint(t);
            const unsigned out = (__ballot_sync(FULL, lt_zero(bx) || gt_pos(bx, __double_as_longlong(glim))) >> base) & 7u;
            const unsigned hb = (__ballot_sync(FULL, th >= 0x3fe00000u && th < 0x7ff00000u) >> base) & 7u;   // t >= 0.5
            const unsigned zf = __shfl_sync(FULL, (lt_pos(bx, __double_as_longlong(Z_RETURN)) ? 1u : 0u) |
                                                      (gt_pos(bx, __double_as_longlong(Z_EXIT)) ? 2u : 0u), base + 2);
            const unsigned near = ((hb & 1u) << 2) | (hb & 2u) | ((hb >> 2) & 1u);
            if (port) {
                const int i = reg - 1;
                uint32_t* cnt = counts + (size_t)i * kNC;
                if (out || ((mask >> near) & 1u)) {
                    reg = R_LOST;
                    if (gl == 0) atomicAdd(cnt + 15, 1u);
                } else if (zf) {
                    // leave (lib.rs:368-385)
                    const double* c = C.mouth[i];
                    if (d < 2) x += c[d] - C.axis;
                    if (zf & 1u) {
                        if (d == 2) x = C.seam + x - Z_RETURN;
                        reg = R_SPLIT;
                        last = i;
                        if (gl == 0) atomicAdd(cnt + 1, 1u);
                    } else {
                        if (d == 2) { x = C.seam - (x - Z_EXIT); v *= -1.0; }
                        reg = R_COMBINE;
                        last = -1;
                        if (gl == 0) { atomicAdd(cnt + 2, 1u); atomicAdd(cnt + 16 + sp, 1u); }
                    }
                    changed = true;
                }
            }
        }
        if (__any_sync(FULL, changed)) {
            enter_region(changed);
            coordinate(changed);
            const double t2 = locate(changed);
            if (changed) t = t2;
        }
        {
            const double omt = 1.0 - t;
            if (gl < 3) { tw[2 * gl] = omt; tw[2 * gl + 1] = t; }
        }
        __syncwarp();
        const bool put = have && (reg >= R_LOST || k >= steps);
        if (__any_sync(FULL, put)) {
            turn = true;
            if (put) {
                if (gl < 3) {
                    (gl == 0 ? T.x : gl == 1 ? T.y : T.z)[id] = x;
                    (gl == 0 ? T.vx : gl == 1 ? T.vy : T.vz)[id] = v;
                }
                if (gl == 0) { T.rng[id] = rng; T.region[id] = reg; T.last[id] = last; }
                have = false;
            }
        }
    }
    if (gl != 0) n_cube = n_port = n_idle = 0;
    add_steps(stepc, n_cube, n_port, n_idle);
}

}  // namespace

struct mq_tandem {
    int dev = 0;
    std::string err;
    mq_tandem_desc desc;
    TConst C;
    std::vector<std::pair<const float*, void*>> bufs;   // host array -> device copy (shared arrays uploaded once)
    void* tr = nullptr;
    size_t tr_cap = 0;
    void* drive = nullptr;
    size_t drive_cap = 0;
    uint32_t* counts = nullptr;
    unsigned long long* stepc = nullptr;   // executed track-steps: cube, driven port, idle port; mixed engine's
                                           // cell-cache fills: cube, port; queue head of the FP64 kernel
    char* stage = nullptr;                 // pinned: a small call's tracks, then the counters
    mqtm::State* mix = nullptr;            // the mixed-precision engine (MQ_PREC_MIXED)
    cudaStream_t st = nullptr;
    cudaEvent_t ev[2] = {nullptr, nullptr};
};

namespace {
mq_status tfail(mq_tandem* t, mq_status c, const std::string& m) {
    if (t) t->err = m;
    return c;
}
#define TCK(call, what) do { cudaError_t c_ = (call); if (c_ != cudaSuccess) return tfail(t, c_ == cudaErrorMemoryAllocation ? MQ_ERR_NOMEM : MQ_ERR_CUDA, std::string(what) + ": " + cudaGetErrorString(c_)); } while (0)
}  // namespace

extern "C" {

mq_status mq_tandem_create(const mq_tandem_desc* d, int32_t device, mq_tandem** out) {
    if (!out) return MQ_ERR_INVALID;
    *out = nullptr;
    if (!d || !d->cube_rf4 || !d->cube_dc4[0] || !d->cube_dc4[1] || d->nspecies < 1 ||
        d->nspecies > 5 || !(d->dt > 0) || !(d->cube_h_mm > 0) ||   // five charge-state counters per port
        (d->precision != MQ_PREC_F64 && d->precision != MQ_PREC_MIXED))
        return MQ_ERR_INVALID;
    for (int a = 0; a < 3; ++a)
        if (d->cube_dims[a] < 2) return MQ_ERR_INVALID;
    for (const mq_tandem_port& p : d->port) {
        if (!p.rf4 || !p.ac4 || !p.dc4 || !p.gate4 || !(p.h > 0)) return MQ_ERR_INVALID;
        for (int a = 0; a < 3; ++a)
            if (p.dims[a] < 2) return MQ_ERR_INVALID;
    }
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || device < 0 || device >= ndev) { cudaGetLastError(); return MQ_ERR_NO_DEVICE; }
    mq_tandem* t = new (std::nothrow) mq_tandem();
    if (!t) return MQ_ERR_NOMEM;
    t->dev = device;
    t->desc = *d;
    auto bail = [&](mq_status s) { mq_tandem_destroy(t); return s; };
    if (cudaSetDevice(device) != cudaSuccess) return bail(MQ_ERR_CUDA);
    if (cudaStreamCreateWithFlags(&t->st, cudaStreamNonBlocking) != cudaSuccess) return bail(MQ_ERR_CUDA);
    for (auto& e : t->ev) if (cudaEventCreate(&e) != cudaSuccess) return bail(MQ_ERR_CUDA);
    // upload a node array (float4 per node) unless the same host array is already resident
    auto upload = [&](const float* src, size_t nodes, const float4** dst) -> bool {
        for (auto& b : t->bufs)
            if (b.first == src) { *dst = static_cast<const float4*>(b.second); return true; }
        void* p = nullptr;
        if (cudaMalloc(&p, nodes * 16) != cudaSuccess) return false;
        t->bufs.emplace_back(src, p);
        if (cudaMemcpy(p, src, nodes * 16, cudaMemcpyHostToDevice) != cudaSuccess) return false;
        *dst = static_cast<const float4*>(p);
        return true;
    };
    TConst& C = t->C;
    std::memset(&C, 0, sizeof(C));
    const size_t cn = (size_t)d->cube_dims[0] * d->cube_dims[1] * d->cube_dims[2];
    if (!upload(d->cube_rf4, cn, &C.crf) || !upload(d->cube_dc4[0], cn, &C.cdc[0]) || !upload(d->cube_dc4[1], cn, &C.cdc[1]))
        return bail(MQ_ERR_NOMEM);
    for (int i = 0; i < 9; ++i) {
        const mq_tandem_port& p = d->port[i];
        TPort& P = C.port[i];
        const size_t kn = (size_t)p.dims[0] * p.dims[1] * p.dims[2];
        if (!upload(p.rf4, kn, &P.rf) || !upload(p.ac4, kn, &P.ac) || !upload(p.dc4, kn, &P.dc) || !upload(p.gate4, kn, &P.gate))
            return bail(MQ_ERR_NOMEM);
        for (int a = 0; a < 3; ++a) {
            P.kn[a] = p.dims[a];
            P.lim[a] = (double)(p.dims[a] - 1) * p.h;   // World::lim (world.rs:145)
        }
        P.kh = p.h;
        P.inv_kh = 1.0 / p.h;
        P.idle = p.tone_khz == 0.0;
    }
    if (cudaMalloc(&t->counts, kTail) != cudaSuccess) return bail(MQ_ERR_NOMEM);
    if (cudaMallocHost(&t->stage, kStageMax + kTail) != cudaSuccess) { cudaGetLastError(); return bail(MQ_ERR_NOMEM); }   // 0.2 ms: not in an advance
    t->stepc = reinterpret_cast<unsigned long long*>(reinterpret_cast<char*>(t->counts) + kCntBytes);
    C.cube = d->cube;
    for (int a = 0; a < 3; ++a) { C.cn[a] = d->cube_dims[a]; C.clo[a] = d->cube_lo_mm[a]; }
    C.ch_mm = d->cube_h_mm;
    C.inv_ch_mm = 1.0 / d->cube_h_mm;
    double mouths[18];
    mq_tandem_layout(d, &C.seam, &C.size, mouths);
    for (int i = 0; i < 9; ++i) { C.mouth[i][0] = mouths[2 * i]; C.mouth[i][1] = mouths[2 * i + 1]; }
    double ent[2];
    mq_cube_port_axis(&d->cube, -1, ent);
    C.ent_b = ent[0]; C.ent_c = ent[1];
    C.axis = d->ch_axis_mm * 1e-3;
    C.ap_r = d->cube.ap_r;
    C.l_ext_m = d->cube.l_ext * 0.001;
    C.dt = d->dt;
    C.gate_v = d->gate_bias_v;
    {   // the FP32 face filter and the range that needs none
        const mq_cube_geom& g = d->cube;
        CubeF& F = C.F;
        F.size = (float)mqc::size(g); F.c0 = (float)mqc::c0(g); F.pitch = (float)g.pitch; F.half_d = (float)(g.d / 2.0);
        F.t_pcb = (float)g.t_pcb; F.gap = (float)g.gap; F.ptd = (float)mqc::post_top_depth(g); F.stem_r = (float)g.stem_r;
        F.clear_r = (float)g.clear_r; F.rod_hole = (float)(g.d / 2.0 + g.rod_clear_extra); F.l_ext = (float)g.l_ext;
        F.cap_reach = (float)(g.l_ext + g.cap_gap); F.cap_r = (float)g.cap_r; F.ap_r = (float)g.ap_r;
        // Coordinates near a surface are at most m, and an FP32 distance of two of them is off by about 10 * 2^-24 m;
        // 2^-17 m is over ten times that. In the cube as built (m = 126 mm) it would be 1 um; 2 um is the least taken.
        const double m = mqc::size(g) + 2.0 * (std::fabs(g.l_ext) + std::fabs(g.cap_gap) + std::fabs(g.cap_r));
        const double near = std::fmax(2e-3, m * 0x1.0p-17);
        F.near = (float)near;
        const double apart = std::fmin(0.499, 0.5 - near / std::fabs(g.pitch));
        F.round_port = (float)apart;
        // Which of two posts is nearer does not matter where both are farther than any radius of theirs, as on the axis
        // of the entrance, where the tracks come in (200,000 of them, 200 steps: 57 ms with the exact test there).
        const double radii = std::fmax(std::fmax(g.d / 2.0, g.stem_r), std::fmax(g.clear_r, g.d / 2.0 + g.rod_clear_extra));
        F.round_post = apart * g.pitch > radii + 4.0 * near ? 1.0f : (float)apart;
        F.ent_b = (float)C.ent_b; F.ent_c = (float)C.ent_c;
        F.n = g.n; F.array = g.array;
        F.ent_axis = g.ent_axis; F.ent_side = g.ent_side; F.ent_cell0 = g.ent_cell[0]; F.ent_cell1 = g.ent_cell[1];
        F.ext_axis = g.ext_axis; F.ext_side = g.ext_side; F.ext_cell0 = g.ext_cell[0]; F.ext_cell1 = g.ext_cell[1];
        auto word = [](double v) {
            int64_t b;
            std::memcpy(&b, &v, 8);
            return (int32_t)(b >> 32);
        };
        const double lo = mqc::post_top_depth(g) + 0.01, hi = mqc::size(g) - lo, zhi = std::fmin(hi, C.seam * 1000.0 - 0.01);
        C.in_lo = word(lo * 1e-3) + 1;
        for (int a = 0; a < 3; ++a) {
            const double top = (a == 2 ? zhi : hi) * 1e-3;
            const int32_t up = top > 0.0 ? word(top) : 0;
            C.in_n[a] = lo > 0.0 && up > C.in_lo ? (uint32_t)(up - C.in_lo) : 0u;
        }
    }
    const double mg = 28.0 * mqp::AMU;
    const double ngas = d->pressure_pa / (mqp::KB * d->temp_k);
    C.s_gas = sqrt(mqp::KB * d->temp_k / mg);
    for (int s = 0; s < d->nspecies; ++s) {   // SpPhys::new (world.rs:342-347)
        const double m = d->species[s].mass * mqp::AMU;
        const double qm = d->species[s].z * mqp::QE / m;
        C.sp[s].qmdt = qm * d->dt;
        C.sp[s].s_ion = sqrt(mqp::KB * d->temp_k / m);
        C.sp[s].mr = mg / (m + mg);
        C.sp[s].nsd = (ngas * (d->species[s].ccs * 1e-20)) * d->dt;
    }
    if (d->precision == MQ_PREC_MIXED) {
        mqtm::DevFields f;
        f.crf = C.crf;
        f.cdc[0] = C.cdc[0];
        f.cdc[1] = C.cdc[1];
        for (int i = 0; i < 9; ++i) {
            f.prf[i] = C.port[i].rf; f.pac[i] = C.port[i].ac; f.pdc[i] = C.port[i].dc; f.pgate[i] = C.port[i].gate;
        }
        std::string err;
        t->mix = mqtm::create(*d, f, t->st, err);
        if (!t->mix) { mq_tandem_destroy(t); return MQ_ERR_NOMEM; }
        if (cudaStreamSynchronize(t->st) != cudaSuccess) return bail(MQ_ERR_CUDA);
    }
    *out = t;
    return MQ_OK;
}

void mq_tandem_destroy(mq_tandem* t) {
    if (!t) return;
    cudaSetDevice(t->dev);
    if (t->st) cudaStreamSynchronize(t->st);
    for (auto& b : t->bufs) cudaFree(b.second);
    if (t->tr) cudaFree(t->tr);
    if (t->drive) cudaFree(t->drive);
    if (t->counts) cudaFree(t->counts);
    if (t->stage) cudaFreeHost(t->stage);
    if (t->mix) mqtm::destroy(t->mix);
    for (auto& e : t->ev) if (e) cudaEventDestroy(e);
    if (t->st) cudaStreamDestroy(t->st);
    delete t;
}

const char* mq_tandem_last_error(mq_tandem* t) { return t ? t->err.c_str() : "null tandem"; }

mq_status mq_tandem_advance(mq_tandem* t, mq_tracks* tr, size_t n, uint64_t step0, uint64_t steps, mq_port_counts counts[9],
                            mq_tandem_stats* stats) {
    if (!t || !tr || !counts) return MQ_ERR_INVALID;
    if (n > 0xFFFFFFF0ull) return tfail(t, MQ_ERR_TOO_LARGE, "at most 2^32-16 tracks");
    TCK(cudaSetDevice(t->dev), "cudaSetDevice");
    const size_t tb = n * (7 * 8 + 3 * 4);
    if (t->tr_cap < tb) {
        if (t->tr) cudaFree(t->tr);
        t->tr = nullptr; t->tr_cap = 0;
        TCK(cudaMalloc(&t->tr, tb ? tb : 16), "track buffers");
        t->tr_cap = tb;
    }
    char* base = static_cast<char*>(t->tr);
    Tracks T;
    void* host[10] = {tr->x, tr->y, tr->z, tr->vx, tr->vy, tr->vz, tr->rng, tr->sp, tr->region, tr->last};
    const size_t sz[10] = {8, 8, 8, 8, 8, 8, 8, 4, 4, 4};
    void* dev[10];
    size_t off = 0;
    for (int k = 0; k < 10; ++k) {
        if (!host[k]) return tfail(t, MQ_ERR_INVALID, "track array missing");
        dev[k] = base + off;
        off += sz[k] * n;
    }
    T.x = (double*)dev[0]; T.y = (double*)dev[1]; T.z = (double*)dev[2];
    T.vx = (double*)dev[3]; T.vy = (double*)dev[4]; T.vz = (double*)dev[5];
    T.rng = (uint64_t*)dev[6]; T.sp = (int32_t*)dev[7]; T.region = (int32_t*)dev[8]; T.last = (int32_t*)dev[9];
    const mqtm::Tracks64 T64{T.x, T.y, T.z, T.vx, T.vy, T.vz, T.rng, T.sp, T.region, T.last};
    for (size_t i = 0; i < n; ++i)   // the kernel indexes species constants and counters by these
        if (tr->sp[i] < 0 || tr->sp[i] >= t->desc.nspecies || tr->region[i] < 0 || tr->region[i] > R_DETECTED ||
            tr->last[i] < -1 || tr->last[i] > 8)
            return tfail(t, MQ_ERR_INVALID, "track " + std::to_string(i) + " has an invalid species, region or last port");
    // Few tracks go through one pinned block, in one copy each way: ten copies of pageable arrays cost
    // 5 us each whatever their size. Many are copied array by array, which the driver does as fast as a
    // host memcpy would stage them; the block holds their counters alone (copied pageable, these cost 30 us).
    const bool staged = tb <= kStageMax;
    TCK(cudaStreamSynchronize(t->st), "tandem");   // a call that failed may have left copies of the block under way
    char* const tail = t->stage + kStageMax;   // port counters, then step counters: their device order
    if (staged) {
        size_t o = 0;
        for (int k = 0; k < 10; ++k) { std::memcpy(t->stage + o, host[k], sz[k] * n); o += sz[k] * n; }
        TCK(cudaMemcpyAsync(base, t->stage, tb, cudaMemcpyHostToDevice, t->st), "track upload");
    } else {
        for (int k = 0; k < 10; ++k) TCK(cudaMemcpyAsync(dev[k], host[k], sz[k] * n, cudaMemcpyHostToDevice, t->st), "track upload");
    }
    for (int i = 0; i < 9; ++i) std::memcpy(tail + (size_t)i * kNC * 4, &counts[i], sizeof(mq_port_counts));
    std::memset(tail + kCntBytes, 0, kTail - kCntBytes);
    TCK(cudaMemcpyAsync(t->counts, tail, kTail, cudaMemcpyHostToDevice, t->st), "counter upload");
    // Drive table: up to kTab steps per upload; kernels of `per` steps each, about 2^27 track-steps
    // per launch so that no single launch runs for long.
    const uint64_t kTab = 65536;
    const uint64_t tab = steps < kTab ? (steps ? steps : 1) : kTab;
    if (t->drive_cap < tab * 10 * 8) {
        if (t->drive) cudaFree(t->drive);
        t->drive = nullptr; t->drive_cap = 0;
        TCK(cudaMalloc(&t->drive, tab * 10 * 8), "drive table");
        t->drive_cap = tab * 10 * 8;
    }
    int sms = 0;
    if (!t->mix) {   // one block of the FP64 kernel per SM: the shared memory asked for lets no second one in
        TCK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, t->dev), "device attributes");
        TCK(cudaFuncSetAttribute(k_tandem<16>, cudaFuncAttributeMaxDynamicSharedMemorySize, kTPad), "tandem kernel");
        TCK(cudaFuncSetAttribute(k_tandem<4>, cudaFuncAttributeMaxDynamicSharedMemorySize, kTPad), "tandem kernel");
    }
    uint64_t per = n ? ((uint64_t)1 << 27) / n : tab;
    per = per < 32 ? 32 : (per > 4096 ? 4096 : per);
    Tones tones;
    tones.f[0] = t->desc.f_rf; tones.v[0] = t->desc.v_rf; tones.dt = t->desc.dt;
    for (int i = 0; i < 9; ++i) { tones.f[1 + i] = t->desc.port[i].tone_khz * 1000.0; tones.v[1 + i] = t->desc.port[i].v_ac; }
    const int forms = t->mix ? mqtm::two_forms(t->mix, *tr, n, steps) : 0;
    uint32_t launches = 0;
    const uint64_t h2d = tb + 9 * kNC * 4;
    for (uint64_t s = 0; s < steps || s == 0; s += tab) {
        const uint64_t k = steps - s < tab ? steps - s : tab;
        if (k) {
            const unsigned blocks = (unsigned)((k * 10 + 127) / 128);
            if (t->mix) k_drive<float><<<blocks, 128, 0, t->st>>>(tones, step0 + s, (uint32_t)k, (float*)t->drive);
            else k_drive<double><<<blocks, 128, 0, t->st>>>(tones, step0 + s, (uint32_t)k, (double*)t->drive);
            TCK(cudaGetLastError(), "drive kernel");
            ++launches;
        }
        if (s == 0) {
            TCK(cudaEventRecord(t->ev[0], t->st), "event");   // times the step kernels (and later table blocks)
            if (t->mix) TCK(mqtm::load(t->mix, T64, (uint32_t)n, t->st, &launches), "mixed tandem load");
        }
        if (!steps) break;
        if (t->mix) {
            TCK(mqtm::run(t->mix, (uint32_t)n, (const float*)t->drive, step0 + s, k, forms, t->counts, t->stepc, t->st, &launches),
                "mixed tandem kernel");
            continue;
        }
        for (uint64_t q = 0; q < k && n; q += per, ++launches) {
            const uint64_t m = k - q < per ? k - q : per;
            uint32_t* head = reinterpret_cast<uint32_t*>(t->stepc + 5);
            TCK(cudaMemsetAsync(head, 0, sizeof(*head), t->st), "queue head");
            if (n <= 8 * (size_t)sms)
                k_tandem<16><<<sms, kTBlock, kTPad, t->st>>>(t->C, T, (uint32_t)n, (const double*)t->drive + q * 10, (uint32_t)m,
                                                             t->counts, t->stepc, head);
            else
                k_tandem<4><<<sms, kTBlock, kTPad, t->st>>>(t->C, T, (uint32_t)n, (const double*)t->drive + q * 10, (uint32_t)m,
                                                            t->counts, t->stepc, head);
            TCK(cudaGetLastError(), "tandem kernel");
        }
    }
    if (t->mix) TCK(mqtm::store(t->mix, T64, (uint32_t)n, t->st, &launches), "mixed tandem store");
    TCK(cudaEventRecord(t->ev[1], t->st), "event");
    if (staged) TCK(cudaMemcpyAsync(t->stage, base, tb, cudaMemcpyDeviceToHost, t->st), "track download");
    else
        for (int k = 0; k < 10; ++k) TCK(cudaMemcpyAsync(host[k], dev[k], sz[k] * n, cudaMemcpyDeviceToHost, t->st), "track download");
    TCK(cudaMemcpyAsync(tail, t->counts, kTail, cudaMemcpyDeviceToHost, t->st), "counter download");
    TCK(cudaStreamSynchronize(t->st), "tandem");
    if (staged) {
        size_t o = 0;
        for (int k = 0; k < 10; ++k) { std::memcpy(host[k], t->stage + o, sz[k] * n); o += sz[k] * n; }
    }
    for (int i = 0; i < 9; ++i) std::memcpy(&counts[i], tail + (size_t)i * kNC * 4, sizeof(mq_port_counts));
    unsigned long long sc[5];
    std::memcpy(sc, tail + kCntBytes, sizeof(sc));
    if (stats) {
        float ms = 0.0f;
        cudaEventElapsedTime(&ms, t->ev[0], t->ev[1]);
        std::memset(stats, 0, sizeof(*stats));
        stats->steps_cube = sc[0];
        stats->steps_port = sc[1];
        stats->steps_idle = sc[2];
        stats->cell_fills_cube = sc[3];
        stats->cell_fills_port = sc[4];
        stats->kernel_ms = ms;
        stats->launches = launches;
        stats->h2d_bytes = h2d;
        stats->d2h_bytes = tb + 9 * kNC * 4 + sizeof(sc);
    }
    return MQ_OK;
}

}  // extern "C"

MQ_CHECK_READER(mq_check_read_tandem)
