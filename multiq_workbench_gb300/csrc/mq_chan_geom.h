// Channel geometry (chsim Geom, simulation/chsim/src/channel.rs:18-120): electrode of a grid node and its
// potential in a basis, for host and device. Evaluated in IEEE double without FMA contraction, so both
// classify a node identically.
#pragma once
#include <math.h>
#include <stdint.h>

#include "mq_grid.h"

#if defined(__CUDACC__)
#define MQG_HD __host__ __device__ inline
#else
#define MQG_HD inline
#endif

namespace mqgeo {

struct Layers { double l[8]; };

MQG_HD Layers layers_of(const mq_geom* g) {
    Layers L;
    double l1 = g->q1_start, l2 = l1 + g->q1_len, l3 = l2 + g->gap, l4 = l3 + g->plate;
    double l5 = l4 + g->gap, l6 = l5 + g->q2_len, l7 = l6 + g->gap, l8 = l7 + g->plate;
    double v[8] = {l1, l2, l3, l4, l5, l6, l7, l8};
    for (int i = 0; i < 8; ++i) L.l[i] = v[i];
    return L;
}

MQG_HD int geom_nz(const mq_geom* g) { return (int)(layers_of(g).l[7] / g->h_mm + 1e-6); }
MQG_HD double geom_center(const mq_geom* g) { return g->coef * g->de / 2.0 + g->de / 2.0; }
MQG_HD double geom_axis(const mq_geom* g) { return (double)(g->n_xy / 2) * g->h_mm; }

// quadrant of (x, y) about the axis; -1 on an axis line (channel.rs:65-67)
MQG_HD int quad(double x, double y, double a) {
    if (x < a && y < a) return 0;
    if (x > a && y < a) return 1;
    if (x < a && y > a) return 2;
    if (x > a && y > a) return 3;
    return -1;
}

// rod membership test of channel.rs:70-79 (rod centre by quadrant and tilt mode)
MQG_HD bool rod_q(const mq_geom* g, double a, double c, double x, double y, double z, double zmid,
           int q, double sq, double d, bool q1) {
    double cx, cy;
    const double s2 = sqrt(2.0);
    if (g->tilt_mode == 0) {
        switch (q) {
            case 0: cx = a - c; cy = a - c + sq; break;
            case 1: cx = a + c; cy = a - c + sq; break;
            case 2: cx = a - c; cy = a + c - sq; break;
            default: cx = a + c; cy = a + c - sq; break;
        }
    } else if (g->tilt_mode == 2) {
        switch (q) {
            case 0: cx = a - c + sq / s2; cy = a - c + sq / s2; break;
            case 1: cx = a + c - sq / s2; cy = a - c + sq / s2; break;
            case 2: cx = a - c + sq / s2; cy = a + c - sq / s2; break;
            default: cx = a + c - sq / s2; cy = a + c - sq / s2; break;
        }
    } else {
        switch (q) {
            case 0: cx = a - c; cy = a - c; break;
            case 1: cx = a + c; cy = a - c; break;
            case 2: cx = a - c + sq; cy = a + c; break;
            default: cx = a + c - sq; cy = a + c; break;
        }
    }
    if (q1) {
        const double* m = g->mis[q];
        cx += m[0] + m[2] * (z - zmid);
        cy += m[1] + m[3] * (z - zmid);
    }
    double dx = x - cx, dy = y - cy;
    return sqrt(dx * dx + dy * dy) < d / 2.0 + g->grow * g->h_mm;
}

enum Kind { K_Q1 = 0, K_STEM3, K_PLATE, K_STEM5, K_Q2, K_STEM7, K_SLAB };
MQG_HD uint8_t code(int kind, int q) { return (uint8_t)(1 + kind * 4 + q); }

// Geom::classify (channel.rs:62-101): electrode code of node (i, j, k), 0 = free.
MQG_HD uint8_t classify(const mq_geom* g, const Layers& L, int i, int j, int k) {
    const double h = g->h_mm;
    const double x = i * h, y = j * h, z = k * h;
    const double a = geom_axis(g), c = geom_center(g);
    const double zmid = g->q1_start + g->q1_len / 2.0;
    const double eps = 1e-9;
    const double l1 = L.l[0], l2 = L.l[1], l3 = L.l[2], l4 = L.l[3], l5 = L.l[4], l6 = L.l[5],
                 l7 = L.l[6], l8 = L.l[7];
    if (z <= l1 + eps) return 0;
    if (z <= l2 + eps) {
        double sq = g->alpha * (l2 - z);
        int q = quad(x, y, a);
        return (q >= 0 && rod_q(g, a, c, x, y, z, zmid, q, sq, g->de, true)) ? code(K_Q1, q) : 0;
    }
    if (z <= l3 + eps) {
        int q = quad(x, y, a);
        return (q >= 0 && rod_q(g, a, c, x, y, z, zmid, q, 0.0, g->stem_d, false)) ? code(K_STEM3, q) : 0;
    }
    if (z <= l4 + eps) {
        double dx = x - a, dy = y - a;
        double r2 = dx * dx + dy * dy;
        double rh = g->hole_d / 2.0 - g->grow * g->h_mm;
        return r2 < rh * rh ? 0 : code(K_PLATE, 0);
    }
    if (z <= l5 + eps) {
        int q = quad(x, y, a);
        return (q >= 0 && rod_q(g, a, c, x, y, z, zmid, q, 0.0, g->stem_d, false)) ? code(K_STEM5, q) : 0;
    }
    if (z <= l6 + eps) {
        double sq = g->q2_flare_bug ? g->alpha * (l2 - z) : 0.0;
        int q = quad(x, y, a);
        return (q >= 0 && rod_q(g, a, c, x, y, z, zmid, q, sq, g->de, false)) ? code(K_Q2, q) : 0;
    }
    if (z <= l7 + eps) {
        int q = quad(x, y, a);
        return (q >= 0 && rod_q(g, a, c, x, y, z, zmid, q, 0.0, g->stem_d, false)) ? code(K_STEM7, q) : 0;
    }
    if (z <= l8 + eps) return code(K_SLAB, 0);
    return 0;
}

MQG_HD double rf_sign(int q) { return (q == 0 || q == 3) ? -1.0 : 1.0; }  // channel.rs:104
MQG_HD double ac_sign(int q) { return (q == 0 || q == 2) ? -1.0 : 1.0; }  // channel.rs:105

// basis_value (channel.rs:111-120) for an electrode code
MQG_HD double basis_value(int basis, uint8_t e, int ac_mode) {
    int kind = (e - 1) / 4, q = (e - 1) % 4;
    switch (basis) {
        case MQ_BASIS_RF:
            return (kind == K_Q1 || kind == K_STEM3 || kind == K_STEM5 || kind == K_Q2 || kind == K_STEM7) ? rf_sign(q) : 0.0;
        case MQ_BASIS_AC:
            if (kind == K_Q1 || kind == K_STEM3) return (ac_mode == 1 && q >= 2) ? 0.0 : ac_sign(q);
            return 0.0;
        case MQ_BASIS_DC_Q1: return (kind == K_Q1 || kind == K_STEM3) ? 1.0 : 0.0;
        case MQ_BASIS_DC_PLATE: return kind == K_PLATE ? 1.0 : 0.0;
        case MQ_BASIS_DC_DOWN: return (kind == K_STEM5 || kind == K_Q2 || kind == K_STEM7 || kind == K_SLAB) ? 1.0 : 0.0;
        default: return 0.0;
    }
}

}  // namespace mqgeo
