// Adjoint of the nonbonded forces and du/dlambda with respect to the per-atom
// parameters (charge, sigma/2, sqrt(epsilon)) and the per-atom w offsets.
//
// For upstream gradients G (of du_dx, [N,3]) and g (of du_dl, scalar) it
// accumulates the vector-Jacobian product
//   dPhi/dtheta,  Phi = sum_i G_i . du_dx_i + g * du_dl,
// pair by pair, recomputing each pair's terms in FP64 from the original
// coordinates and parameters (nothing is stored by the forward pass). It walks
// the same tile list and scaled-pair list as the forward kernels.
//
// Per pair (r = x_i - x_j minimum image, dw = w_i - w_j,
// w = cutoff * (plane + offset * lambda), d^2 = r.r + dw^2 < cutoff^2) the
// energy is U(d) = s * [cs * q_i q_j erfc(beta d)/d + ls * 4 e_i e_j ((S/d)^12 - (S/d)^6)]
// (S = sig_i + sig_j; s = +1 for all pairs, -1 for the scaled exclusions;
// LJ only where e_i e_j != 0), as timemachine/potentials/nonbonded.py:29-59,
// 133-264 define it. With h = U'(d)/d the pair adds h r to du_dx_i, -h r to
// du_dx_j and h dw cutoff (off_i - off_j) to du_dl, so
//   Phi_pair = h * B,  B = (G_i - G_j).r + g * dw * cutoff * (off_i - off_j),
//   dPhi/dp      = B * dh/dp                         (p: q, sig, eps of i or j)
//   dPhi/doff_i  = B * h'(d) * dw * cutoff * lambda / d
//                  + g * h * cutoff * (cutoff * lambda * (off_i - off_j) + dw)
//   dPhi/doff_j  = -(the same).
// The derivatives of erfc(beta d)/d follow from d/dd erfc(beta d) =
// -2 beta / sqrt(pi) exp(-beta^2 d^2).
#pragma once

#include "nb_kernels.cuh"

namespace tmb {

struct AdjointArgs {
    int N;
    int S;
    const double *x;      // [N,3]
    const double *p;      // [N,3]
    const double *box;    // [9]
    const int *plane;     // [N]
    const int *offset;    // [N]
    double lambda, beta, cutoff;
    const unsigned *perm; // [S] slot -> atom
    const unsigned *tile_cols;
    const int4 *items;
    int M;
    const int *pair_idxs; // [M,2] atoms
    const double *scales; // [M,2]
    double pair_sign;     // -1: the listed pairs are subtracted (exclusions), +1: added
    const double *g_dx;   // [N,3]
    double g_dl;          // upstream gradient of du_dl,
    const double *g_dl_at; // or where it lies on the device (nullptr: g_dl)
    double *grad_p; // [N,3] +=
    double *grad_w; // [N] +=
    DevState *state;
};

// What the pair terms need of one atom: coordinates, parameters (q, sigma/2,
// sqrt eps), the upstream gradient of its du_dx, and its lambda plane/offset.
struct AdjAtom {
    double x[3];
    double p[3];
    double g[3];
    int plane;
    int offset;
};

__device__ __forceinline__ AdjAtom load_adj_atom(const AdjointArgs &a, int atom) {
    AdjAtom t;
    for (int d = 0; d < 3; d++) {
        t.x[d] = a.x[3 * (size_t)atom + d];
        t.p[d] = a.p[3 * (size_t)atom + d];
        t.g[d] = a.g_dx[3 * (size_t)atom + d];
    }
    t.plane = a.plane[atom];
    t.offset = a.offset[atom];
    return t;
}

// Gradient contributions of one pair: to atom i (q, sig, eps, off) and atom j.
struct PairGrad {
    double qi, si, ei, wi;
    double qj, sj, ej, wj;
};

// One pair within the cutoff: r = x_i - x_j (minimum image), dw and doff the
// differences of w and of the offsets, G the difference of the upstream
// gradients.
__device__ __forceinline__ PairGrad adjoint_terms(
    const AdjointArgs &a, const double (&r)[3], const double d2, const double dw, const double doff,
    const double (&pi)[3], const double (&pj)[3], const double (&G)[3], const double g_dl, double cs, double ls,
    double sign) {
    PairGrad out;
    const double c = a.cutoff;
    const double d = sqrt(d2);
    const double inv_d = 1.0 / d;
    const double qi = pi[0], si = pi[1], ei = pi[2];
    const double qj = pj[0], sj = pj[1], ej = pj[2];

    // electrostatics: E = erfc(beta d)/d
    const double bd = a.beta * d;
    const double g0 = erfc(bd);
    const double g1 = -2.0 * a.beta * 0.56418958354775628695 * exp(-bd * bd); // d erfc(beta d)/dd
    const double g2 = -2.0 * a.beta * a.beta * d * g1;                           // second derivative
    const double E1 = g1 * inv_d - g0 * inv_d * inv_d;
    const double E2 = g2 * inv_d - 2.0 * g1 * inv_d * inv_d + 2.0 * g0 * inv_d * inv_d * inv_d;
    double h = cs * qi * qj * E1 * inv_d;
    double hp = cs * qi * qj * (E2 * inv_d - E1 * inv_d * inv_d);
    double dh_qi = cs * qj * E1 * inv_d, dh_qj = cs * qi * E1 * inv_d;
    double dh_s = 0, dh_ei = 0, dh_ej = 0;
    if (ei * ej != 0) {
        const double S = si + sj;
        const double sd = S * inv_d;
        const double sd6 = sd * sd * sd * sd * sd * sd;
        const double inv_d2 = inv_d * inv_d;
        // U_lj = 4 e e (sd^12 - sd^6); h_lj = U'/d = 4 e e (-12 sd^12 + 6 sd^6) / d^2
        const double base = (-12.0 * sd6 * sd6 + 6.0 * sd6) * inv_d2;
        const double ee = 4.0 * ls * ei * ej;
        h += ee * base;
        hp += ee * (168.0 * sd6 * sd6 - 48.0 * sd6) * inv_d2 * inv_d;
        dh_s = ee * (-144.0 * sd6 * sd6 + 36.0 * sd6) * inv_d2 / S;
        dh_ei = 4.0 * ls * ej * base;
        dh_ej = 4.0 * ls * ei * base;
    }
    h *= sign;
    hp *= sign;
    const double B = G[0] * r[0] + G[1] * r[1] + G[2] * r[2] + g_dl * dw * c * doff;
    out.qi = sign * B * dh_qi;
    out.qj = sign * B * dh_qj;
    out.si = sign * B * dh_s;
    out.sj = out.si;
    out.ei = sign * B * dh_ei;
    out.ej = sign * B * dh_ej;
    const double dphi_doff_i = B * hp * dw * c * a.lambda * inv_d + g_dl * h * c * (c * a.lambda * doff + dw);
    out.wi = dphi_doff_i;
    out.wj = -dphi_doff_i;
    return out;
}

__device__ __forceinline__ void adjoint_add(const AdjointArgs &a, int atom, double q, double s, double e, double w) {
    atomicAdd(a.grad_p + 3 * (size_t)atom + 0, q);
    atomicAdd(a.grad_p + 3 * (size_t)atom + 1, s);
    atomicAdd(a.grad_p + 3 * (size_t)atom + 2, e);
    atomicAdd(a.grad_w + atom, w);
}

// A scaled pair.
__device__ __forceinline__ PairGrad
adjoint_pair(const AdjointArgs &a, const AdjAtom &I, const AdjAtom &J, double g_dl, double cs, double ls, double sign) {
    double r[3], G[3];
    double r2 = 0;
    for (int d = 0; d < 3; d++) {
        const double L = a.box[4 * d];
        double v = I.x[d] - J.x[d];
        v -= L * floor(v / L + 0.5);
        r[d] = v;
        r2 += v * v;
        G[d] = I.g[d] - J.g[d];
    }
    const double c = a.cutoff;
    const double doff = (double)(I.offset - J.offset);
    const double dw = c * ((I.plane - J.plane) + doff * a.lambda);
    const double d2 = r2 + dw * dw;
    if (!(d2 < c * c)) {
        return {0, 0, 0, 0, 0, 0, 0, 0};
    }
    return adjoint_terms(a, r, d2, dw, doff, I.p, J.p, G, g_dl, cs, ls, sign);
}

constexpr int ADJ_WARPS = 4;

// The RG rows of a tile, one instance per warp, and their gradient sums: one
// copy per RG-lane group, as in the forward tile walk (nb_kernels.cuh).
template <int RG> struct AdjRows {
    double x[3][RG];
    double p[3][RG];
    double g[3][RG];
    int plane[RG];
    int offset[RG];
    double lo[3], hi[3]; // smallest and largest row coordinates
    double acc[4][TILE]; // q, sig, eps, offset: [copy * RG + row]
};

// One warp per tile, walked as the forward pair kernel walks it: lane l owns
// column l (atom and sums in registers), marks the rows within the cutoff,
// then takes its marked rows one per step, all lanes with the pair arithmetic
// at once. FP64 arithmetic bounds the kernel (erfc, exp, the divisions), so what
// matters is that the lanes of a step hold pairs: 0.8 of them do, against 0.4
// when every row met every column (96 -> 67 us per launch at 5,000 atoms on
// B200). Row sums are FP64 atomics in shared memory
// (zero terms, most sig, eps and offset ones, are not added), columns' and rows'
// totals one global FP64 atomic each per tile. The scaled pairs follow as one
// lane per pair. Dynamic work counter state->next_item (reset by the staging).
template <int RG> static __global__ void __launch_bounds__(ADJ_WARPS * 32) k_adjoint(AdjointArgs a) {
    __shared__ AdjRows<RG> rows_sm[ADJ_WARPS];
    if (a.state->error) {
        return;
    }
    AdjRows<RG> &sm = rows_sm[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31;
    const unsigned S = (unsigned)a.S;
    const int chunk = max(1, a.state->items_chunk); // the list's, whichever call built it
    const int n_tile_units = a.tile_cols ? a.state->n_items * chunk : 0;
    const int n_total = n_tile_units + (a.M + TILE - 1) / TILE;
    const double L[3] = {a.box[0], a.box[4], a.box[8]};
    const double inv_L[3] = {1.0 / L[0], 1.0 / L[1], 1.0 / L[2]};
    const double c = a.cutoff;
    const double g_dl = a.g_dl_at ? *a.g_dl_at : a.g_dl;
    const int rot = lane & (RG - 1);
    const int copy = lane & ~(RG - 1);
    for (int k = 0; k < 4; k++) {
        sm.acc[k][lane] = 0.0;
    }
    for (;;) {
        int unit = 0;
        if (lane == 0) {
            unit = atomicAdd(&a.state->next_item, 1);
        }
        unit = __shfl_sync(FULL_MASK, unit, 0);
        if (unit >= n_total) {
            break;
        }
        if (unit >= n_tile_units) {
            const int pair = (unit - n_tile_units) * TILE + lane;
            if (pair < a.M) {
                const int ai = a.pair_idxs[2 * pair], aj = a.pair_idxs[2 * pair + 1];
                const PairGrad g = adjoint_pair(
                    a, load_adj_atom(a, ai), load_adj_atom(a, aj), g_dl, a.scales[2 * pair], a.scales[2 * pair + 1],
                    a.pair_sign);
                adjoint_add(a, ai, g.qi, g.si, g.ei, g.wi);
                adjoint_add(a, aj, g.qj, g.sj, g.ej, g.wj);
            }
            continue;
        }
        const int4 it = a.items[unit / chunk];
        const int t = unit - (unit / chunk) * chunk;
        if (t >= it.z) {
            continue; // warp-uniform
        }
        const unsigned row_first = (unsigned)(it.x * RG);
        const unsigned i = row_first + rot;
        const unsigned j = a.tile_cols[((long long)it.y + t) * TILE + lane];
        const int ai = i < S ? (int)a.perm[i] : -1;
        const int aj = j < S ? (int)a.perm[j] : -1;
        AdjAtom I = {}, J = {};
        if (ai >= 0) {
            I = load_adj_atom(a, ai);
        }
        if (aj >= 0) {
            J = load_adj_atom(a, aj);
        }
        const double nan = __longlong_as_double(0x7fffffffffffffffll);
        for (int d = 0; d < 3; d++) {
            // rows past the last: NaN coordinates, which fmin / fmax pass over
            // and no cutoff test passes
            double v = ai >= 0 ? I.x[d] : nan;
            if (lane < RG) {
                sm.x[d][lane] = v;
                sm.p[d][lane] = I.p[d];
                sm.g[d][lane] = I.g[d];
            }
            double lo = v, hi = v;
#pragma unroll
            for (int o = RG / 2; o > 0; o >>= 1) {
                lo = fmin(lo, __shfl_xor_sync(FULL_MASK, lo, o));
                hi = fmax(hi, __shfl_xor_sync(FULL_MASK, hi, o));
            }
            if (lane == 0) {
                sm.lo[d] = lo;
                sm.hi[d] = hi;
            }
        }
        if (lane < RG) {
            sm.plane[lane] = I.plane;
            sm.offset[lane] = I.offset;
        }
        __syncwarp();
        const bool alch = __any_sync(FULL_MASK, I.plane != 0 || I.offset != 0 || J.plane != 0 || J.offset != 0);
        // the column's image against the rows: one shift where the smallest and
        // the largest row coordinate give the same count
        double shift[3];
        bool one_image = true;
        for (int d = 0; d < 3; d++) {
            const double n = floor((sm.lo[d] - J.x[d]) * inv_L[d] + 0.5);
            one_image = one_image && n == floor((sm.hi[d] - J.x[d]) * inv_L[d] + 0.5);
            shift[d] = -L[d] * n;
        }
        const bool wrap = __any_sync(FULL_MASK, aj >= 0 && !one_image);
        auto displacement = [&](int row, double (&r)[3]) {
            double r2 = 0;
            for (int d = 0; d < 3; d++) {
                double v = sm.x[d][row] - J.x[d];
                v = wrap ? v - L[d] * floor(v * inv_L[d] + 0.5) : v + shift[d];
                r[d] = v;
                r2 += v * v;
            }
            return r2;
        };
        auto w_difference = [&](int row, double &doff) {
            doff = (double)(sm.offset[row] - J.offset);
            return c * ((sm.plane[row] - J.plane) + doff * a.lambda);
        };
        unsigned mask = 0;
#pragma unroll 4
        for (int row = 0; row < RG; row++) {
            double r[3], doff;
            double d2 = displacement(row, r);
            if (alch) {
                const double dw = w_difference(row, doff);
                d2 += dw * dw;
            }
            mask |= d2 < c * c ? 1u << row : 0u;
        }
        // a column of the row group itself pairs with the rows before it
        const unsigned own = j - row_first;
        mask &= aj < 0 ? 0u : (own < (unsigned)RG ? (1u << own) - 1 : FULL_MASK);
        unsigned m = RG == TILE ? __funnelshift_r(mask, mask, rot)
                                : ((mask | (mask << (RG & 31))) >> rot) & (unsigned)((1ull << RG) - 1);
        double cq = 0, csig = 0, ceps = 0, cw = 0;
        for (unsigned n = __reduce_max_sync(FULL_MASK, (unsigned)__popc(m)); n > 0; n--) {
            if (m == 0) {
                continue;
            }
            const int row = (__ffs(m) - 1 + rot) & (RG - 1);
            m &= m - 1;
            double r[3], doff = 0, dw = 0;
            double d2 = displacement(row, r);
            if (alch) {
                dw = w_difference(row, doff);
                d2 += dw * dw;
            }
            const double pi[3] = {sm.p[0][row], sm.p[1][row], sm.p[2][row]};
            const double G[3] = {sm.g[0][row] - J.g[0], sm.g[1][row] - J.g[1], sm.g[2][row] - J.g[2]};
            const PairGrad g = adjoint_terms(a, r, d2, dw, doff, pi, J.p, G, g_dl, 1.0, 1.0, 1.0);
            cq += g.qj;
            csig += g.sj;
            ceps += g.ej;
            cw += g.wj;
            const double terms[4] = {g.qi, g.si, g.ei, g.wi};
            for (int k = 0; k < 4; k++) {
                if (terms[k] != 0) {
                    atomicAdd(&sm.acc[k][copy + row], terms[k]);
                }
            }
        }
        __syncwarp();
        for (int k = 0; k < 4; k++) {
            double v = sm.acc[k][lane];
            sm.acc[k][lane] = 0.0;
#pragma unroll
            for (int o = RG; o < TILE; o <<= 1) {
                v += __shfl_xor_sync(FULL_MASK, v, o);
            }
            if (lane < RG && ai >= 0 && v != 0) {
                atomicAdd(k < 3 ? a.grad_p + 3 * (size_t)ai + k : a.grad_w + ai, v);
            }
            const double w = k == 0 ? cq : k == 1 ? csig : k == 2 ? ceps : cw;
            if (aj >= 0 && w != 0) {
                atomicAdd(k < 3 ? a.grad_p + 3 * (size_t)aj + k : a.grad_w + aj, w);
            }
        }
        __syncwarp();
    }
}

} // namespace tmb
