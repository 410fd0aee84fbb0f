// Device pipeline of one nonbonded evaluation on sm_100a.
//
// Per evaluation (stream-ordered, no host synchronisation):
//   k_check_prepare   rebuild decision (any atom moved > padding/2, or box
//                     changed), box validation, and the per-slot FP32 staging
//                     of coordinates, w, parameters (and dp/dlambda) using the
//                     current slot order.
//   k_order_slots / k_stage_blocks / k_build_tiles
//                     neighbour-list rebuild: slot order, staging of the new
//                     order, tiles; every one returns at once unless the
//                     rebuild flag is set, so the sequence is graph-capturable.
//                     k_build_tiles clears the accumulators in any case.
//                     (k_prepare_sort: the whole front of a small system's call;
//                     k_bin_keys / k_bin_scan / k_bin_scatter: the order of many atoms.)
//   k_pair            persistent kernel over the tile work items and the
//                     exclusion / scaled-pair chunks (dynamic scheduling).
//   k_finalize        scatter of the slot-ordered int64 accumulators into the
//                     caller's original-order outputs.
//
// The work of each stage follows the reference pipeline
// (timemachine/cpp/src/nonbonded_all_pairs.cu:222-433,
//  timemachine/cpp/src/neighborlist.cu:126-185,
//  timemachine/cpp/src/nonbonded_pair_list.cu:95-166); the data layout,
// spatial sort, scheduling and fusion are this file's own.
//
// The non-template kernels have internal linkage (static), so that several
// translation units can include this file.
#pragma once

#include "nb_pair_math.cuh"
#include "tmnb.h"

namespace tmb {

constexpr unsigned FULL_MASK = 0xffffffffu;
constexpr int TILE = 32;

// Sticky device-side state of one potential instance.
struct DevState {
    int rebuild;          // 1: the neighbour list must be rebuilt in this evaluation
    int error;            // sticky error code (TMNB_ERR_* values), 0 = ok
    int n_items;          // tile work items produced by the last rebuild
    int next_item;        // dynamic work counter of k_pair (reset by k_check_prepare, or in a
                          // fused MD step by the integrator kernel that staged the coordinates)
    unsigned done_ctas;   // completion counter of k_build_tiles
    unsigned total_tiles; // tiles produced by the last rebuild
    int rebuilds;         // number of rebuilds performed (diagnostics)
    int n_dep;            // lambda-dependent tiles listed by k_dep_tiles (multi-window calls)
    int dep_dirty;        // 1: the list of lambda-dependent tiles must be redone (rebuild, or lamdep changed)
    int items_chunk;      // tiles per work item in the list of the last rebuild
    int item_count;       // work items reserved so far by the rebuild in progress (0 between rebuilds)
    int plain_until;      // rebuilds before this one keep the plain order (site_order)
};

// Error codes written into DevState::error (mirrored in include/tmnb.h).
constexpr int DEV_ERR_NONORTHO_BOX = 3;
constexpr int DEV_ERR_BOX_TOO_SMALL = 4;

// Up to this many lambda windows are evaluated together (one launch sequence).
constexpr int MAX_WINDOWS = TMNB_MAX_WINDOWS;

struct SlotArrays {
    float4 *posw;            // [K][S] x, y, z, w(lambda_k)
    float4 *prm;             // [K][S] q, sig, eps, dw/dlambda (parameters at lambda_k)
    float4 *dprm;            // [K][S] dq/dl, dsig/dl, deps/dl, 0 (interpolated only)
    unsigned char *lamdep;   // [S] 1 when the atom's staged values depend on lambda
    // FP64 pair arithmetic only (nullptr otherwise): the same values unrounded
    double4 *posw64;         // [K][S]
    double4 *prm64;          // [K][S]
    double4 *dprm64;         // [K][S] (interpolated only)
};

// One lambda window as the staging sees it: the values f(lambda) and
// derivatives g = df/dlambda of the four lambda transforms (charge, sigma,
// epsilon, w) of timemachine/cpp/src/kernels/k_lambda_transformer_jit.cuh:8-22,
// evaluated on the host for each call (identity transform: f = lambda, g = 1).
struct LambdaWindow {
    double f_q, g_q;
    double f_s, g_s;
    double f_e, g_e;
    double f_w, g_w;
};

struct PrepareArgs {
    int N;                      // atoms in the system
    int S;                      // slots (atoms in the evaluated set)
    const double *x;            // [N,3]
    const double *p;            // [N,3] or [2N,3] (interpolated)
    const double *box;          // [3,3]
    int K;                      // lambda windows
    LambdaWindow lam[MAX_WINDOWS];
    double cutoff;
    double padding;
    const int *plane;           // [N]
    const int *offset;          // [N]
    int interpolated;
    SlotArrays slots;
};

// Staging of one atom for window k, with the transforms of window k:
// w = cutoff*(plane + offset*f_w), dw/dlambda = offset*g_w*cutoff
// (timemachine/cpp/src/kernels/k_lambda_transformer_jit.cuh:25-55);
// interpolated parameters p = (1-f) p0 + f p1 and dp/dlambda = g (p1 - p0)
// per parameter column (same file :57-98). v[0..5] receives the staged
// parameters and their lambda derivatives in FP64.
__device__ __forceinline__ void window_values(const PrepareArgs &a, int atom, int k, double &w, double &dw_dl,
                                              double (&v)[6]) {
    const int plane = a.plane[atom];
    const int offset = a.offset[atom];
    const LambdaWindow &L = a.lam[k];
    w = (plane + offset * L.f_w) * a.cutoff;
    dw_dl = offset * L.g_w * a.cutoff;
    const double *p0 = a.p + 3 * (size_t)atom;
    v[0] = p0[0];
    v[1] = p0[1];
    v[2] = p0[2];
    v[3] = v[4] = v[5] = 0.0;
    if (a.interpolated) {
        const double *p1 = a.p + 3 * ((size_t)a.N + atom);
        v[0] = (1 - L.f_q) * p0[0] + L.f_q * p1[0];
        v[1] = (1 - L.f_s) * p0[1] + L.f_s * p1[1];
        v[2] = (1 - L.f_e) * p0[2] + L.f_e * p1[2];
        v[3] = L.g_q * (p1[0] - p0[0]);
        v[4] = L.g_s * (p1[1] - p0[1]);
        v[5] = L.g_e * (p1[2] - p0[2]);
    }
}

__device__ __forceinline__ void stage_window(const PrepareArgs &a, int s, int atom, int k) {
    double w, dw_dl, v[6];
    window_values(a, atom, k, w, dw_dl, v);
    const double *xa = a.x + 3 * (size_t)atom;
    const size_t o = (size_t)k * a.S + s;
    a.slots.posw[o] = make_float4((float)xa[0], (float)xa[1], (float)xa[2], (float)w);
    a.slots.prm[o] = make_float4((float)v[0], (float)v[1], (float)v[2], (float)dw_dl);
    if (a.interpolated) {
        a.slots.dprm[o] = make_float4((float)v[3], (float)v[4], (float)v[5], 0.0f);
    }
    if (a.slots.posw64 != nullptr) {
        a.slots.posw64[o] = make_double4(xa[0], xa[1], xa[2], w);
        a.slots.prm64[o] = make_double4(v[0], v[1], v[2], dw_dl);
        if (a.interpolated) {
            a.slots.dprm64[o] = make_double4(v[3], v[4], v[5], 0.0);
        }
    }
}

// An atom is lambda-dependent when its offset is nonzero, its end states
// differ, or any window stages parameter values other than window 0's: pairs
// of lambda-independent atoms give the same per-pair values in every window,
// bit for bit.
__device__ __forceinline__ bool lambda_dependent(const PrepareArgs &a, int atom) {
    if (a.offset[atom] != 0) {
        return true;
    }
    if (!a.interpolated) {
        return false;
    }
    const double *p0 = a.p + 3 * (size_t)atom;
    const double *p1 = a.p + 3 * ((size_t)a.N + atom);
    if (p0[0] != p1[0] || p0[1] != p1[1] || p0[2] != p1[2]) {
        return true;
    }
    double w, dw_dl, first[6], v[6];
    window_values(a, atom, 0, w, dw_dl, first);
    for (int k = 1; k < a.K; k++) {
        window_values(a, atom, k, w, dw_dl, v);
        for (int c = 0; c < 6; c++) {
            if (v[c] != first[c]) {
                return true;
            }
        }
    }
    return false;
}

// Stage one atom into its slot for every window and record its lambda dependence.
__device__ __forceinline__ void prepare_slot(const PrepareArgs &a, int s, int atom) {
    for (int k = 0; k < a.K; k++) {
        stage_window(a, s, atom, k);
    }
    a.slots.lamdep[s] = lambda_dependent(a, atom) ? 1 : 0;
}

// ---------------------------------------------------------------------------
// Rebuild decision + staging.
// ---------------------------------------------------------------------------
// The work of thread tid of n_threads.
__device__ __forceinline__ void check_prepare(
    const PrepareArgs &a,
    const unsigned *perm, // [S] slot -> atom
    const double *nb_x,   // [N,3] coordinates at the last rebuild (nullptr: no neighbour list)
    const double *nb_box, // [9]
    DevState *state,
    const int tid,
    const int n_threads) {
    if (tid == 0) {
        state->next_item = 0;
        if (nb_x != nullptr) {
            // Orthorhombic box whose every edge is at least twice cutoff+padding
            // (timemachine/cpp/src/nonbonded_all_pairs.cu:315-329); checked in
            // the reference's order, so an off-diagonal entry wins.
            const double db_cutoff = (a.cutoff + a.padding) * 2;
            int err = 0;
            for (int k = 0; k < 9 && err == 0; k++) {
                if (k == 0 || k == 4 || k == 8) {
                    if (a.box[k] < db_cutoff) {
                        err = DEV_ERR_BOX_TOO_SMALL;
                    }
                } else if (a.box[k] != 0.0) {
                    err = DEV_ERR_NONORTHO_BOX;
                }
            }
            if (err != 0) {
                state->error = err;
            }
            for (int k = 0; k < 9; k++) {
                if (a.box[k] != nb_box[k]) {
                    state->rebuild = 1;
                }
            }
        }
    }
    // one thread per (window, slot), slots fastest: the K windows' staging
    // stores spread over the grid; the window-0 thread of a slot also takes
    // the rebuild test and the slot's lambda dependence
    const double half_pad2 = 0.25 * a.padding * a.padding;
    const size_t total = (size_t)a.S * (size_t)a.K;
    for (size_t t = tid; t < total; t += n_threads) {
        const int k = (int)(t / (size_t)a.S);
        const int s = (int)(t - (size_t)k * a.S);
        const int atom = perm[s];
        stage_window(a, s, atom, k);
        if (k != 0) {
            continue;
        }
        if (nb_x != nullptr) {
            const double *xn = a.x + 3 * (size_t)atom;
            const double *xo = nb_x + 3 * (size_t)atom;
            const double dx = xn[0] - xo[0];
            const double dy = xn[1] - xo[1];
            const double dz = xn[2] - xo[2];
            if (moved_beyond_half_padding(dx, dy, dz, half_pad2)) {
                state->rebuild = 1; // benign race: every writer stores 1
            }
        }
        const unsigned char dep = lambda_dependent(a, atom) ? 1 : 0;
        if (a.slots.lamdep[s] != dep) {
            a.slots.lamdep[s] = dep;
            // the lambda-dependent tiles change with it (benign race: every writer stores the same)
            state->dep_dirty = 1;
            state->n_dep = 0;
        }
    }
}

static __global__ void k_check_prepare(
    PrepareArgs a,
    const unsigned *__restrict__ perm,
    const double *__restrict__ nb_x,
    const double *__restrict__ nb_box,
    DevState *state) {
    grid_dependency_wait();
    check_prepare(
        a, perm, nb_x, nb_box, state, blockIdx.x * blockDim.x + threadIdx.x, (int)(gridDim.x * blockDim.x));
}

// ---------------------------------------------------------------------------
// Spatial sort: atoms are binned into a 2^b x 2^b x 2^b grid whose cells are
// ordered along a 3D Hilbert curve; a counting sort over the cells gives the
// slot order. The Hilbert index uses Skilling's transposed-axes algorithm
// (J. Skilling, "Programming the Hilbert curve", AIP Conf. Proc. 707, 2004).
// Order inside a cell is arbitrary: results do not depend on it because all
// accumulation is exact integer arithmetic.
// ---------------------------------------------------------------------------
__device__ __forceinline__ unsigned hilbert_index_3d(unsigned x, unsigned y, unsigned z, int bits) {
    unsigned X[3] = {x, y, z};
    const unsigned M = 1u << (bits - 1);
    for (unsigned Q = M; Q > 1; Q >>= 1) {
        const unsigned P = Q - 1;
        for (int i = 0; i < 3; i++) {
            if (X[i] & Q) {
                X[0] ^= P;
            } else {
                const unsigned t = (X[0] ^ X[i]) & P;
                X[0] ^= t;
                X[i] ^= t;
            }
        }
    }
    X[1] ^= X[0];
    X[2] ^= X[1];
    unsigned t = 0;
    for (unsigned Q = M; Q > 1; Q >>= 1) {
        if (X[2] & Q) {
            t ^= Q - 1;
        }
    }
    X[0] ^= t;
    X[1] ^= t;
    X[2] ^= t;
    unsigned h = 0;
    for (int b = bits - 1; b >= 0; b--) {
        h = (h << 3) | (((X[0] >> b) & 1u) << 2) | (((X[1] >> b) & 1u) << 1) | ((X[2] >> b) & 1u);
    }
    return h;
}

// Atoms with a lambda offset take the first slots, in the order of their indices
// (a ligand's follow its bonds), as long as their row groups stay compact. A group
// with atoms of two places goes through the columns around both, and the rebuild
// waits for its one CTA. The tile build measures the groups: when the half diagonal
// of one's box exceeds SITE_EXTENT cutoffs, the next SITE_RETRY rebuilds keep the
// plain order, and then the rule is tried again. Measured on B200 at 22,840 atoms,
// us per call with a rebuild, those atoms first wherever they are / plain order / this
// rule: forces, one ligand 130 / 128 / 130, with a distant ion 167 / 129 / 128, two
// ligands 162 / 129 / 129, 1 % of the atoms anywhere 163 / 133 / 132; 12 windows (more
// than one such atom in 128: first wherever they are) 189 / 198 / 189, 227 / 202 / 203,
// 226 / 214 / 214, 274 / 391 / 274.
constexpr unsigned SITE_KEY = 0xffffffffu; // instead of a cell's
constexpr float SITE_EXTENT = 1.0f;
constexpr int SITE_RETRY = 1000;

struct SortArgs {
    int N;
    int S;
    const double *x;
    const double *box;
    const int *set_atoms; // [S] atoms of the evaluated set, nullptr: identity (S == N)
    int n_first;          // set entries [0, n_first) sort before the others (interaction
                          // group rows before columns); S: one group
    const int *offset;     // [N] lambda offsets: atoms with one may take the first slots
                           // (nullptr: no such rule)
    const int *site_atoms; // [n_site] those atoms
    int n_site;
    bool site_always; // whatever the extent of their row groups
    int grid_bits;        // b: 2^b cells per axis
    int hilbert;          // 0: keep the set order
    unsigned *keys;       // [S]
    int *bin_count;       // [8^b]
    int *bin_cursor;      // [8^b]
};

__device__ __forceinline__ int set_atom(const SortArgs &a, int k) { return a.set_atoms ? a.set_atoms[k] : k; }

// Position of an atom's cell on the curve.
__device__ __forceinline__ unsigned cell_key(const SortArgs &a, int atom) {
    const int G = 1 << a.grid_bits;
    unsigned c[3];
    for (int d = 0; d < 3; d++) {
        const double L = a.box[d * 4];
        double v = a.x[3 * (size_t)atom + d];
        v -= L * floor(v / L);
        int ci = (int)(v / L * G);
        ci = ci < 0 ? 0 : (ci >= G ? G - 1 : ci);
        c[d] = (unsigned)ci;
    }
    return hilbert_index_3d(c[0], c[1], c[2], a.grid_bits);
}

// Whether the site's atoms come first in this rebuild: not in the ones after a wide
// row group. The same for every thread until the tile build has ended.
__device__ __forceinline__ bool site_order(const DevState *state) {
    const volatile DevState *now = state;
    return now->rebuilds >= now->plain_until;
}
__device__ __forceinline__ bool site_first(const SortArgs &a, const DevState *state) {
    return a.offset != nullptr && (a.site_always || site_order(state));
}
// The cell at which the curve starts: next to the last site atom, so that the row
// group which holds it is compact too.
__device__ __forceinline__ unsigned first_cell(const SortArgs &a, const bool site) {
    return site ? cell_key(a, a.site_atoms[a.n_site - 1]) : 0u;
}

__device__ __forceinline__ void bin_key(const SortArgs &a, int k, const bool site, const unsigned first) {
    {
        const int atom = set_atom(a, k);
        if (site && a.offset[atom] != 0) {
            a.keys[k] = SITE_KEY;
            return;
        }
        unsigned key = cell_key(a, atom);
        if (k >= a.n_first) {
            key += 1u << (3 * a.grid_bits);
        }
        if (site) { // once round the curve, whose ends are neighbours across the periodic boundary
            key = (key - first) & ((1u << (3 * a.grid_bits)) - 1);
        }
        a.keys[k] = key;
        atomicAdd(&a.bin_count[key], 1);
    }
}

static __global__ void k_bin_keys(SortArgs a, const DevState *state) {
    grid_dependency_wait();
    if (!state->rebuild || state->error || !a.hilbert) {
        return;
    }
    const bool site = site_first(a, state);
    const unsigned first = first_cell(a, site);
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < a.S; k += gridDim.x * blockDim.x) {
        bin_key(a, k, site, first);
    }
}

// Single-CTA exclusive scan of the cell counts (and reset of the counts and
// of the tile-build counters).
__device__ __forceinline__ void bin_scan_cta(const SortArgs &a, DevState *state) {
    if (threadIdx.x == 0) {
        state->done_ctas = 0;
        state->total_tiles = 0;
    }
    if (!a.hilbert) {
        return;
    }
    const int NB = (1 << (3 * a.grid_bits)) * (a.n_first < a.S ? 2 : 1);
    __shared__ int warp_sums[32];
    __shared__ int carry;
    if (threadIdx.x == 0) {
        carry = site_first(a, state) ? a.n_site : 0;
    }
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const int wid = threadIdx.x >> 5;
    const int nwarps = blockDim.x >> 5;
    // four consecutive cells per thread (NB is a multiple of 64, the counts
    // 256-byte aligned): a quarter of the passes and barriers
    for (int base = 0; base < NB; base += 4 * (int)blockDim.x) {
        const int b = base + 4 * (int)threadIdx.x;
        const int4 c4 = b < NB ? *reinterpret_cast<const int4 *>(a.bin_count + b) : make_int4(0, 0, 0, 0);
        const int v = c4.x + c4.y + c4.z + c4.w;
        int incl = v;
        for (int o = 1; o < 32; o <<= 1) {
            const int n = __shfl_up_sync(FULL_MASK, incl, o);
            if (lane >= o) {
                incl += n;
            }
        }
        if (lane == 31) {
            warp_sums[wid] = incl;
        }
        __syncthreads();
        if (wid == 0) {
            int ws = lane < nwarps ? warp_sums[lane] : 0;
            for (int o = 1; o < 32; o <<= 1) {
                const int n = __shfl_up_sync(FULL_MASK, ws, o);
                if (lane >= o) {
                    ws += n;
                }
            }
            if (lane < nwarps) {
                warp_sums[lane] = ws; // inclusive
            }
        }
        __syncthreads();
        const int warp_prefix = wid > 0 ? warp_sums[wid - 1] : 0;
        if (b < NB) {
            const int e = carry + warp_prefix + incl - v;
            *reinterpret_cast<int4 *>(a.bin_cursor + b) = make_int4(e, e + c4.x, e + c4.x + c4.y, e + c4.x + c4.y + c4.z);
            *reinterpret_cast<int4 *>(a.bin_count + b) = make_int4(0, 0, 0, 0);
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            carry += warp_sums[nwarps - 1];
        }
        __syncthreads();
    }
}

static __global__ void k_bin_scan(SortArgs a, DevState *state) {
    grid_dependency_wait();
    if (!state->rebuild || state->error) {
        return;
    }
    bin_scan_cta(a, state);
}

// Slot of set entry k after the counting sort; records the slot order and the
// coordinates of the rebuild.
__device__ __forceinline__ int scatter_slot(
    const SortArgs &sa, int k, unsigned *__restrict__ perm, int *__restrict__ slot_of, double *__restrict__ nb_x) {
    const int atom = set_atom(sa, k);
    const int s = sa.hilbert ? atomicAdd(&sa.bin_cursor[sa.keys[k]], 1) : k;
    perm[s] = (unsigned)atom;
    if (slot_of) {
        slot_of[atom] = s;
    }
    nb_x[3 * (size_t)atom + 0] = sa.x[3 * (size_t)atom + 0];
    nb_x[3 * (size_t)atom + 1] = sa.x[3 * (size_t)atom + 1];
    nb_x[3 * (size_t)atom + 2] = sa.x[3 * (size_t)atom + 2];
    return s;
}

// Slot order after the counting sort (the site's atoms, then the cells in
// Hilbert order, arbitrary within a cell), or the set order without the sort.
__device__ __forceinline__ void order_slot(const SortArgs &sa, int k, const bool site, unsigned *perm) {
    if (!sa.hilbert) {
        perm[k] = (unsigned)set_atom(sa, k);
        return;
    }
    if (site && k < sa.n_site) {
        perm[k] = (unsigned)sa.site_atoms[k];
    }
    const unsigned key = sa.keys[k];
    if (key != SITE_KEY) {
        perm[atomicAdd(&sa.bin_cursor[key], 1)] = (unsigned)set_atom(sa, k);
    }
}

static __global__ void k_bin_scatter(SortArgs sa, unsigned *perm, const DevState *state) {
    grid_dependency_wait();
    if (!state->rebuild || state->error) {
        return;
    }
    const bool site = site_first(sa, state);
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < sa.S; k += gridDim.x * blockDim.x) {
        order_slot(sa, k, site, perm);
    }
}

__device__ __forceinline__ float wrap_delta(float d, float L, float inv_L) { return d - L * rintf(d * inv_L); }

// What the atoms of a block are imaged next to: its first atom's coordinate (any
// other where that one is infinite or NaN, else the whole block would be lost with it).
__device__ __forceinline__ float box_reference(float first) { return fabsf(first) < 3.0e38f ? first : 0.f; }

// Bounding box of the 32-slot block rb (one warp) from its atoms' positions p.
__device__ __forceinline__ void block_bounds_warp(
    const bool valid, const float4 p, const double *box, int rb, float4 *bb_ctr, float4 *bb_ext) {
    const int lane = threadIdx.x & 31;
    const float Lx = (float)box[0], Ly = (float)box[4], Lz = (float)box[8];
    const float iLx = 1.0f / Lx, iLy = 1.0f / Ly, iLz = 1.0f / Lz;
    {
        const float rx = box_reference(__shfl_sync(FULL_MASK, p.x, 0));
        const float ry = box_reference(__shfl_sync(FULL_MASK, p.y, 0));
        const float rz = box_reference(__shfl_sync(FULL_MASK, p.z, 0));
        float dx = wrap_delta(p.x - rx, Lx, iLx);
        float dy = wrap_delta(p.y - ry, Ly, iLy);
        float dz = wrap_delta(p.z - rz, Lz, iLz);
        float mnx = valid ? dx : 3.0e38f, mny = valid ? dy : 3.0e38f, mnz = valid ? dz : 3.0e38f;
        float mxx = valid ? dx : -3.0e38f, mxy = valid ? dy : -3.0e38f, mxz = valid ? dz : -3.0e38f;
        for (int o = 16; o > 0; o >>= 1) {
            mnx = fminf(mnx, __shfl_xor_sync(FULL_MASK, mnx, o));
            mny = fminf(mny, __shfl_xor_sync(FULL_MASK, mny, o));
            mnz = fminf(mnz, __shfl_xor_sync(FULL_MASK, mnz, o));
            mxx = fmaxf(mxx, __shfl_xor_sync(FULL_MASK, mxx, o));
            mxy = fmaxf(mxy, __shfl_xor_sync(FULL_MASK, mxy, o));
            mxz = fmaxf(mxz, __shfl_xor_sync(FULL_MASK, mxz, o));
        }
        if (lane == 0) {
            bb_ctr[rb] = make_float4(rx + 0.5f * (mnx + mxx), ry + 0.5f * (mny + mxy), rz + 0.5f * (mnz + mxz), 0.f);
            // widen by a relative rounding allowance so the box test stays conservative
            bb_ext[rb] = make_float4(
                0.5f * (mxx - mnx) * 1.000001f + 1e-6f,
                0.5f * (mxy - mny) * 1.000001f + 1e-6f,
                0.5f * (mxz - mnz) * 1.000001f + 1e-6f,
                0.f);
        }
    }
}

struct SortTargets {
    unsigned *perm; // [S] slot -> atom
    int *slot_of;   // [N] atom -> slot (nullptr: not needed)
    double *nb_x;   // [N,3] coordinates of the rebuild
    double *nb_box; // [9]
    float4 *bb_ctr, *bb_ext;
    int rows;
};

// The new slot order's 32-slot block rb (one warp): Lennard-Jones atoms first
// within each row group (`rows` slots), then the atoms' staging, the rebuild's
// coordinates and the block's bounding box. With LJ rows first and LJ columns
// in tiles of their own the pair kernel's LJ part runs in fewer steps; sorting
// within row groups, not across them, keeps each group spatially compact.
// Blocks that straddle the interaction group's row/column boundary keep their
// order.
__device__ __forceinline__ void stage_block(
    const SortArgs &sa, const PrepareArgs &pa, const SortTargets &to, const int rb) {
    const int lane = threadIdx.x & 31;
    const int s = rb * TILE + lane;
    const bool valid = s < sa.S;
    const unsigned atom = valid ? to.perm[s] : 0u;
    bool lj = false;
    if (valid) {
        lj = pa.p[3 * (size_t)atom + 2] != 0.0;
        if (pa.interpolated) {
            lj = lj || pa.p[3 * ((size_t)pa.N + atom) + 2] != 0.0;
        }
    }
    const unsigned m = __ballot_sync(FULL_MASK, lj);
    const unsigned vm = __ballot_sync(FULL_MASK, valid);
    int pos = lane;
    if (!(rb * TILE < sa.n_first && min(sa.S, rb * TILE + TILE) > sa.n_first)) {
        const unsigned lt = (1u << lane) - 1u;
        const int seg = lane / to.rows;
        const unsigned segm = (to.rows == TILE ? FULL_MASK : ((1u << to.rows) - 1u)) << (seg * to.rows);
        pos = seg * to.rows + (lj ? __popc(m & lt & segm) : __popc(m & segm) + __popc(vm & ~m & lt & segm));
    }
    __syncwarp(); // every lane has read its slot
    float4 at = make_float4(0.f, 0.f, 0.f, 0.f);
    if (valid) {
        const int ns = rb * TILE + pos;
        to.perm[ns] = atom;
        if (to.slot_of) {
            to.slot_of[atom] = ns;
        }
        const double *xa = pa.x + 3 * (size_t)atom;
        at = make_float4((float)xa[0], (float)xa[1], (float)xa[2], 0.f);
        for (int d = 0; d < 3; d++) {
            to.nb_x[3 * (size_t)atom + d] = xa[d];
        }
        prepare_slot(pa, ns, (int)atom);
    }
    block_bounds_warp(valid, at, sa.box, rb, to.bb_ctr, to.bb_ext);
}

static __global__ void k_stage_blocks(SortArgs sa, PrepareArgs pa, SortTargets to, const DevState *state) {
    grid_dependency_wait();
    if (!state->rebuild || state->error) {
        return;
    }
    const int tid = blockIdx.x * blockDim.x + threadIdx.x;
    if (tid < 9) {
        to.nb_box[tid] = sa.box[tid];
    }
    const int RB = (sa.S + TILE - 1) / TILE;
    for (int rb = tid >> 5; rb < RB; rb += (gridDim.x * blockDim.x) >> 5) {
        stage_block(sa, pa, to, rb);
    }
}

// The slot order (keys, scan, scatter) by one cluster of CTAs with hardware
// barriers between the phases: one launch instead of three, which every call
// that does not rebuild pays for too. Eight SMs are enough for a few ten
// thousand atoms (NonbondedPotential::CLUSTER_SORT_MAX).
constexpr int SORT_CTAS = 8; // the portable cluster size
constexpr int SORT_THREADS = 1024;

// Barrier of the cluster; global memory written before it is visible after it.
__device__ __forceinline__ void cluster_barrier() {
    __threadfence();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

__device__ __forceinline__ void order_slots_cluster(const SortArgs &sa, unsigned *perm, DevState *state) {
    const int tid = blockIdx.x * blockDim.x + threadIdx.x;
    constexpr int T = SORT_CTAS * SORT_THREADS;
    const bool site = site_first(sa, state);
    if (sa.hilbert) {
        const unsigned first = first_cell(sa, site);
        for (int k = tid; k < sa.S; k += T) {
            bin_key(sa, k, site, first);
        }
    }
    cluster_barrier();
    if (blockIdx.x == 0) {
        bin_scan_cta(sa, state);
    }
    cluster_barrier();
    for (int k = tid; k < sa.S; k += T) {
        order_slot(sa, k, site, perm);
    }
}

static __global__ void __cluster_dims__(SORT_CTAS, 1, 1) __launch_bounds__(SORT_THREADS, 1)
    k_order_slots(SortArgs sa, unsigned *perm, DevState *state) {
    grid_dependency_wait();
    if (!state->rebuild || state->error) { // the same for every CTA: nothing here changes them
        return;
    }
    order_slots_cluster(sa, perm, state);
}

// Rebuild decision and staging (k_check_prepare), and where a rebuild is due
// the sort and the new order's staging, by the same cluster: one launch for the
// whole front of a small system's call.
static __global__ void __cluster_dims__(SORT_CTAS, 1, 1) __launch_bounds__(SORT_THREADS, 1)
    k_prepare_sort(SortArgs sa, PrepareArgs pa, SortTargets to, DevState *state) {
    grid_dependency_wait();
    const int tid = blockIdx.x * blockDim.x + threadIdx.x;
    check_prepare(pa, to.perm, to.nb_x, to.nb_box, state, tid, SORT_CTAS * SORT_THREADS);
    cluster_barrier();
    const volatile DevState *now = state;
    if (!now->rebuild || now->error) {
        return;
    }
    order_slots_cluster(sa, to.perm, state);
    cluster_barrier();
    if (tid < 9) {
        to.nb_box[tid] = sa.box[tid];
    }
    const int RB = (sa.S + TILE - 1) / TILE;
    for (int rb = tid >> 5; rb < RB; rb += (SORT_CTAS * SORT_THREADS) >> 5) {
        stage_block(sa, pa, to, rb);
    }
}

// ---------------------------------------------------------------------------
// Tile list. Rows come in groups of `rows` (32, 16 or 8) consecutive slots;
// one CTA (TB_WARPS warps) per row group g. For every 32-slot column block from
// the one holding the group's first slot on (upper triangle) whose bounding
// box is within the list radius of the group's box, each column atom at or
// after the group's first slot is kept when any row atom lies within the list
// radius (minimum image, 3D). Kept atoms are sorted (lambda-dependent atoms
// first, then Lennard-Jones atoms, each by the number of row atoms within the
// cutoff, most first) and packed 32 to a tile, so a tile is rows x 32 pairs and
// its columns have about equally many pairs, which is what the pair kernel's
// lanes wait for (of the lane steps of a 22,840-atom water box 0.80 hold a
// pair, 0.52 with the columns in slot order). The lambda-dependent columns
// share tiles, so fewer tiles are evaluated once per window, and most tiles
// without Lennard-Jones columns skip that part. Smaller row groups sit in
// smaller regions and list fewer out-of-range column atoms. The tiles of row group g occupy a fixed range
// (tile_base) sized by the column blocks it can reach. Each group's CTA cuts
// its tiles into work items of at most `chunk` tiles, written at a range it
// reserves from a counter; the last CTA to finish publishes the item count.
// (Same selection rule as timemachine/cpp/src/kernels/k_neighborlist.cuh:168-427,
// which uses 32-atom row blocks.)
// ---------------------------------------------------------------------------
struct TileArgs {
    int S;
    int RB;           // blocks of 32 slots = ceil(S/32) (column blocks)
    int rows;         // slots per row group: 32, 16 or 8
    int group;        // 1: interaction group (rows [0, row_end) x columns [col_begin, S))
    int row_end;      // S, or the number of row atoms
    int col_begin;    // 0, or the number of row atoms
    int n_row_blocks; // row groups: ceil(row_end/rows)
    int cb_first;     // group: first column block (col_begin/32)
    float radius;     // list radius (cutoff + padding + margin)
    float cutoff;     // the column order counts the row atoms within it
    int n_site;       // atoms that site_first may put into the first slots
    const double *box;
    const float4 *posw;
    const float4 *prm;           // staged parameters (eps in .z)
    const unsigned char *lamdep; // [S] lambda dependence of the slots' atoms
    const float4 *bb_ctr;
    const float4 *bb_ext;
    unsigned *tile_cols;   // [capacity*32] slot of each column atom (S = empty)
    int *rb_ntiles;        // [n_row_blocks] tiles of each row group
    int4 *items;           // [item_capacity] (row group, first tile, tile count, 0)
    int chunk;             // tiles per work item
};

__host__ __device__ __forceinline__ long long tile_offset(int rb, int RB) {
    return (long long)rb * RB - ((long long)rb * (rb - 1)) / 2;
}

// First tile of row group g. Upper triangle: the group reaches the RB - b
// column blocks from its own block b = g*rows/32 on, one tile per block at
// most; with m = 32/rows groups per block that sums to
// m * tile_offset(b, RB) + (g mod m) * (RB - b). Interaction group:
// RB - cb_first tiles per row group.
__host__ __device__ __forceinline__ long long tile_base_rows(int g, int rows, int RB, int group, int cb_first) {
    if (group) {
        return (long long)g * (RB - cb_first);
    }
    const int m = TILE / rows;
    const int b = g / m;
    return (long long)m * tile_offset(b, RB) + (long long)(g - b * m) * (RB - b);
}
__host__ __device__ __forceinline__ long long tile_base(const TileArgs &a, int g) {
    return tile_base_rows(g, a.rows, a.RB, a.group, a.cb_first);
}

constexpr int TB_WARPS = 8;
// Column atoms of a group that the CTA sorts into its tiles; the ones found after
// them follow in the order they were found. Groups of 16 rows list up to 2,000 at 100
// atoms per nm^3 and 1.2 nm, up to 3,500 at 1.6 nm. Measured on B200, us of an energy
// call with a rebuild, 5,000 atoms at 1.6 nm: 78 (doing such a group again, in rounds
// of 32 column blocks, 106; room for 4,608 columns 80); 20,000 atoms 150 (195; 151).
constexpr int TB_COLS = 3072;
constexpr int TB_WINDOWS = 16; // box tests per thread before the atoms are gone through
// sort keys: lambda dependence x Lennard-Jones x 33 row counts
constexpr int TB_KEYS = 2 * 2 * 33;
// Tile-build CTAs per SM the compiler must fit (40 registers; 5 CTAs at 48
// measured the same). The build is bound by instruction issue (ncu at 98,000
// atoms: 75 % of issue slots), so what counts is what it does per column atom:
// measured on B200, us of a forces call with a rebuild, testing every atom of a
// passing block with three barriers per window of 256 blocks -> the atoms in
// reach only, box tests of 16 windows at a time: 98,000 atoms 431 -> 397,
// 22,840 137 -> 130. Loading the next block's atoms ahead: 434.
#ifndef TMNB_TB_CTAS
#define TMNB_TB_CTAS 6
#endif

struct TileBuildSmem {
    // row positions: element pair m holds rows 2m, 2m + 1 (NaN past the group's last)
    alignas(8) float row_x[TILE];
    alignas(8) float row_y[TILE];
    alignas(8) float row_z[TILE];
    float4 row_box[2]; // the row group's box: centre, half-extent
    unsigned cols[TB_COLS];
    unsigned char keys[TB_COLS];
    int bins[TB_KEYS]; // columns of each key, then the next position of each key
    int n_cols; // all of the group's
    float4 queue[TB_WARPS][2 * TILE]; // column atoms in reach of the group's box: position, slot
    unsigned passing[TB_WINDOWS * TB_WARPS]; // column blocks that pass the box test, one bit each
    int is_last;
};

// Writes the group's n columns as tiles from dst on: the collected ones sorted by
// key; those after them are there already. The last tile is padded with S.
// Returns the tiles.
__device__ __forceinline__ int tb_emit(TileBuildSmem &sm, const TileArgs &a, const int n, unsigned *dst) {
    const int lane = threadIdx.x & 31;
    if (threadIdx.x < TILE) {
        constexpr int PER = (TB_KEYS + TILE - 1) / TILE;
        int c[PER], sum = 0;
        for (int k = 0; k < PER; k++) {
            const int b = lane * PER + k;
            c[k] = b < TB_KEYS ? sm.bins[b] : 0;
            sum += c[k];
        }
        int incl = sum;
        for (int o = 1; o < TILE; o <<= 1) {
            const int v = __shfl_up_sync(FULL_MASK, incl, o);
            incl += lane >= o ? v : 0;
        }
        int at = incl - sum;
        for (int k = 0; k < PER; k++) {
            const int b = lane * PER + k;
            if (b < TB_KEYS) {
                sm.bins[b] = at;
            }
            at += c[k];
        }
    }
    __syncthreads();
    for (int k = threadIdx.x; k < min(n, TB_COLS); k += TB_WARPS * 32) {
        dst[atomicAdd(&sm.bins[sm.keys[k]], 1)] = sm.cols[k];
    }
    const int n_out = (n + TILE - 1) / TILE * TILE;
    if (n + (int)threadIdx.x < n_out) {
        dst[n + threadIdx.x] = (unsigned)a.S;
    }
    __syncthreads();
    return n_out / TILE;
}

// Up to 32 column atoms (one per lane, `active`; slot in q.w) against the row
// atoms: those within the list radius of one are collected with their key, or go
// to their place among the group's columns (dst) where TB_COLS are collected.
__device__ __forceinline__ void tb_test_columns(
    TileBuildSmem &sm, const TileArgs &a, const float4 q, const bool active, const bool shifted, const float r2,
    const float Lx, const float Ly, const float Lz, const float iLx, const float iLy, const float iLz,
    unsigned *dst) {
    const int lane = threadIdx.x & 31;
    const float rc2 = a.cutoff * a.cutoff;
    float d2_min = 3.0e38f;
    int near = 0; // row atoms within the cutoff
    // two rows per packed FP32x2 test; a NaN row passes no comparison
    const float2 qx = f2(q.x), qy = f2(q.y), qz = f2(q.z);
    const float2 *rx2 = reinterpret_cast<const float2 *>(sm.row_x);
    const float2 *ry2 = reinterpret_cast<const float2 *>(sm.row_y);
    const float2 *rz2 = reinterpret_cast<const float2 *>(sm.row_z);
    auto test = [&](const float2 dx, const float2 dy, const float2 dz) {
        const float2 d2 = ffma2(dz, dz, ffma2(dy, dy, fmul2(dx, dx)));
        d2_min = fminf(d2_min, fminf(d2.x, d2.y));
        near += d2.x < rc2 ? 1 : 0;
        near += d2.y < rc2 ? 1 : 0;
    };
    if (shifted) {
        for (int r0 = 0; r0 < a.rows / 2; r0 += 4) {
#pragma unroll
            for (int r = r0; r < r0 + 4; r++) {
                test(fsub2(rx2[r], qx), fsub2(ry2[r], qy), fsub2(rz2[r], qz));
            }
        }
    } else {
        const float2 lx = f2(-Lx), ly = f2(-Ly), lz = f2(-Lz), ix = f2(iLx), iy = f2(iLy), iz = f2(iLz);
        for (int r = 0; r < a.rows / 2; r++) {
            test(min_image2(fsub2(rx2[r], qx), lx, ix), min_image2(fsub2(ry2[r], qy), ly, iy),
                 min_image2(fsub2(rz2[r], qz), lz, iz));
        }
    }
    const bool hit = active && d2_min < r2;
    const unsigned hmask = __ballot_sync(FULL_MASK, hit);
    if (hmask == 0) {
        return;
    }
    int at = 0;
    if (lane == 0) {
        at = atomicAdd(&sm.n_cols, __popc(hmask));
    }
    at = __shfl_sync(FULL_MASK, at, 0) + __popc(hmask & ((1u << lane) - 1));
    const int s = __float_as_int(q.w);
    if (hit && at >= TB_COLS) {
        dst[at] = (unsigned)s;
    } else if (hit) {
        const int key = (a.lamdep[s] ? 0 : 66) + (a.prm[s].z != 0.f ? 0 : 33) + 32 - near;
        sm.cols[at] = (unsigned)s;
        sm.keys[at] = (unsigned char)key;
        atomicAdd(&sm.bins[key], 1);
    }
}

__device__ __forceinline__ void build_tiles_cta(const TileArgs &a, const int rb, DevState *state) {
    __shared__ TileBuildSmem sm;

    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const int S = a.S;
    const float Lx = (float)a.box[0], Ly = (float)a.box[4], Lz = (float)a.box[8];
    const float iLx = 1.0f / Lx, iLy = 1.0f / Ly, iLz = 1.0f / Lz;
    const float r2 = a.radius * a.radius;
    const float r2_box = (a.radius + 1e-4f) * (a.radius + 1e-4f);
    const int rows = a.rows;
    const int row_first = rb * rows;
    const int row_n = min(rows, a.row_end - row_first);
    if (warp == 0) {
        // the row group's box, as block_bounds_warp computes a 32-slot block's
        const bool valid = lane < row_n;
        const float4 p = valid ? a.posw[row_first + lane] : make_float4(0.f, 0.f, 0.f, 0.f);
        const float rx = box_reference(__shfl_sync(FULL_MASK, p.x, 0));
        const float ry = box_reference(__shfl_sync(FULL_MASK, p.y, 0));
        const float rz = box_reference(__shfl_sync(FULL_MASK, p.z, 0));
        const float dx = wrap_delta(p.x - rx, Lx, iLx);
        const float dy = wrap_delta(p.y - ry, Ly, iLy);
        const float dz = wrap_delta(p.z - rz, Lz, iLz);
        float mnx = valid ? dx : 3.0e38f, mny = valid ? dy : 3.0e38f, mnz = valid ? dz : 3.0e38f;
        float mxx = valid ? dx : -3.0e38f, mxy = valid ? dy : -3.0e38f, mxz = valid ? dz : -3.0e38f;
        for (int o = 16; o > 0; o >>= 1) {
            mnx = fminf(mnx, __shfl_xor_sync(FULL_MASK, mnx, o));
            mny = fminf(mny, __shfl_xor_sync(FULL_MASK, mny, o));
            mnz = fminf(mnz, __shfl_xor_sync(FULL_MASK, mnz, o));
            mxx = fmaxf(mxx, __shfl_xor_sync(FULL_MASK, mxx, o));
            mxy = fmaxf(mxy, __shfl_xor_sync(FULL_MASK, mxy, o));
            mxz = fmaxf(mxz, __shfl_xor_sync(FULL_MASK, mxz, o));
        }
        if (lane == 0) {
            sm.row_box[0] = make_float4(rx + 0.5f * (mnx + mxx), ry + 0.5f * (mny + mxy), rz + 0.5f * (mnz + mxz), 0.f);
            sm.row_box[1] = make_float4(
                0.5f * (mxx - mnx) * 1.000001f + 1e-6f, 0.5f * (mxy - mny) * 1.000001f + 1e-6f,
                0.5f * (mxz - mnz) * 1.000001f + 1e-6f, 0.f);
            const float ex = mxx - mnx, ey = mxy - mny, ez = mxz - mnz;
            const float widest = 2.0f * SITE_EXTENT * a.cutoff;
            if (row_first < a.n_site && ex * ex + ey * ey + ez * ez > widest * widest &&
                site_order(state)) {
                state->plain_until = state->rebuilds + 1 + SITE_RETRY;
            }
        }
    }
    __syncthreads();
    const float4 rc = sm.row_box[0];
    const float4 re = sm.row_box[1];

    // Row atoms are imaged next to the row block's centre. When every box
    // edge satisfies L/2 - extent >= radius, a column atom imaged next to the
    // centre (once) is at its minimum image from every row atom whenever that
    // distance is below the radius, so the per-pair test needs no wrapping.
    const bool shifted = 0.5f * Lx - re.x >= a.radius + 1e-3f && 0.5f * Ly - re.y >= a.radius + 1e-3f &&
                         0.5f * Lz - re.z >= a.radius + 1e-3f;
    if (threadIdx.x < rows) {
        const int s = row_first + threadIdx.x;
        float4 p = s < a.row_end ? a.posw[s] : make_float4(rc.x, rc.y, rc.z, 0.f);
        p.x = rc.x + wrap_delta(p.x - rc.x, Lx, iLx);
        p.y = rc.y + wrap_delta(p.y - rc.y, Ly, iLy);
        p.z = rc.z + wrap_delta(p.z - rc.z, Lz, iLz);
        sm.row_x[threadIdx.x] = (int)threadIdx.x < row_n ? p.x : __int_as_float(0x7fffffff);
        sm.row_y[threadIdx.x] = p.y;
        sm.row_z[threadIdx.x] = p.z;
    }
    for (int k = threadIdx.x; k < TB_KEYS; k += TB_WARPS * 32) {
        sm.bins[k] = 0;
    }
    if (threadIdx.x == 0) {
        sm.n_cols = 0;
    }
    __syncthreads();
    const int col_lo = a.group ? a.col_begin : row_first; // first column slot of the group's pairs
    const long long base_tile = tile_base(a, rb);
    const unsigned lane_lt = (1u << lane) - 1;

    // The box tests (one column block per thread) leave a bit per block, then
    // warp w goes through the set bits w, w + 8, w + 16 and w + 24 of every word:
    // passing blocks cluster at nearby indices, so interleaving gives every warp
    // about as many, without ranking them.
    const int first_block = a.group ? a.cb_first : row_first / TILE;
    unsigned *const dst = a.tile_cols + base_tile * TILE;
    constexpr int PASS = TB_WINDOWS * TB_WARPS * TILE;
    for (int c0 = first_block; c0 < a.RB; c0 += PASS) {
        const int c_end = min(a.RB, c0 + PASS);
        const int windows = (c_end - c0 + TB_WARPS * TILE - 1) / (TB_WARPS * TILE);
        for (int i = 0; i < windows; i++) {
            const int cb = c0 + i * TB_WARPS * TILE + (int)threadIdx.x;
            bool pass = false;
            if (cb < c_end) {
                const float4 cc = a.bb_ctr[cb];
                const float4 ce = a.bb_ext[cb];
                const float dx = fmaxf(0.f, fabsf(wrap_delta(rc.x - cc.x, Lx, iLx)) - re.x - ce.x);
                const float dy = fmaxf(0.f, fabsf(wrap_delta(rc.y - cc.y, Ly, iLy)) - re.y - ce.y);
                const float dz = fmaxf(0.f, fabsf(wrap_delta(rc.z - cc.z, Lz, iLz)) - re.z - ce.z);
                pass = dx * dx + dy * dy + dz * dz < r2;
            }
            const unsigned m = __ballot_sync(FULL_MASK, pass);
            if (lane == 0) {
                sm.passing[i * TB_WARPS + warp] = m;
            }
        }
        __syncthreads();
        int queued = 0; // atoms in the warp's queue
        for (int b0 = 0; b0 < windows * TB_WARPS; b0 += TILE) {
            const unsigned mine =
                b0 + lane < windows * TB_WARPS ? sm.passing[b0 + lane] & (0x01010101u << warp) : 0u;
            unsigned words = __ballot_sync(FULL_MASK, mine != 0);
            int word = 0;
            for (unsigned m = 0; m != 0 || words != 0; m &= m - 1) {
                if (m == 0) {
                    word = __ffs(words) - 1;
                    words &= words - 1;
                    m = __shfl_sync(FULL_MASK, mine, word);
                }
                const int s = (c0 + (b0 + word) * TILE + __ffs(m) - 1) * TILE + lane;
                const bool valid = s < S;
                const float4 pj = valid ? a.posw[s] : make_float4(0.f, 0.f, 0.f, 0.f);
                // an atom farther than the radius from the row block's box is
                // farther than the radius from every row atom (widened test,
                // conservative under rounding): skip its per-row test
                const float wx = wrap_delta(pj.x - rc.x, Lx, iLx);
                const float wy = wrap_delta(pj.y - rc.y, Ly, iLy);
                const float wz = wrap_delta(pj.z - rc.z, Lz, iLz);
                const float bx = fmaxf(0.f, fabsf(wx) - re.x);
                const float by = fmaxf(0.f, fabsf(wy) - re.y);
                const float bz = fmaxf(0.f, fabsf(wz) - re.z);
                const bool need = valid && s >= col_lo && bx * bx + by * by + bz * bz < r2_box;
                // only the atoms in reach of the box (about half of a block)
                // go on to the row tests, 32 at a time
                const unsigned nmask = __ballot_sync(FULL_MASK, need);
                if (need) {
                    sm.queue[warp][queued + __popc(nmask & lane_lt)] =
                        make_float4(rc.x + wx, rc.y + wy, rc.z + wz, __int_as_float(s));
                }
                queued += __popc(nmask);
                if (queued >= TILE) {
                    __syncwarp();
                    tb_test_columns(sm, a, sm.queue[warp][lane], true, shifted, r2, Lx, Ly, Lz, iLx, iLy, iLz, dst);
                    queued -= TILE;
                    const float4 rest = sm.queue[warp][TILE + lane];
                    __syncwarp();
                    sm.queue[warp][lane] = rest;
                    __syncwarp();
                }
            }
        }
        __syncwarp();
        if (queued > 0) {
            tb_test_columns(sm, a, sm.queue[warp][lane], lane < queued, shifted, r2, Lx, Ly, Lz, iLx, iLy, iLz, dst);
        }
        __syncthreads(); // `passing` is written by the next pass, n_cols read below
    }
    const int tiles = tb_emit(sm, a, sm.n_cols, dst);
    if (warp == 0) {
        const int total = tiles;
        // the group's work items, at a range reserved from the list's
        // counter (items are in any order: the pair kernel schedules them
        // dynamically and its sums do not depend on the order)
        const int ni = (total + a.chunk - 1) / a.chunk;
        int first_item = 0;
        if (lane == 0) {
            a.rb_ntiles[rb] = total;
            atomicAdd(&state->total_tiles, (unsigned)total);
            first_item = atomicAdd(&state->item_count, ni);
        }
        first_item = __shfl_sync(FULL_MASK, first_item, 0);
        const long long first_tile = tile_base(a, rb);
        for (int c = lane; c < ni; c += TILE) {
            const int first = c * a.chunk;
            a.items[first_item + c] = make_int4(rb, (int)(first_tile + first), min(a.chunk, total - first), 0);
        }
    }
    // the last CTA to finish publishes the list
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        const unsigned prev = atomicAdd(&state->done_ctas, 1u);
        sm.is_last = (prev == (unsigned)a.n_row_blocks - 1);
    }
    __syncthreads();
    if (!sm.is_last) {
        return;
    }
    if (threadIdx.x == 0) {
        __threadfence();
        state->n_items = *((volatile int *)&state->item_count);
        state->item_count = 0;
        state->items_chunk = a.chunk;
        state->dep_dirty = 1; // the lambda-dependent tiles follow the new list
        state->n_dep = 0;
        state->rebuilds += 1;
        state->done_ctas = 0;
        state->rebuild = 0;
    }
}

static __global__ void __launch_bounds__(TB_WARPS * 32, TMNB_TB_CTAS) k_build_tiles(
    TileArgs a, unsigned long long *clear, size_t n_clear, DevState *state) {
    grid_dependency_wait();
    // the accumulators the pair kernel adds into, cleared in this launch
    // instead of one of its own
    for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < n_clear; k += (size_t)gridDim.x * blockDim.x) {
        clear[k] = 0;
    }
    if (!state->rebuild || state->error || (int)blockIdx.x >= a.n_row_blocks) {
        return;
    }
    build_tiles_cta(a, blockIdx.x, state);
}

// ---------------------------------------------------------------------------
// Pair kernel.
// ---------------------------------------------------------------------------
struct Accum {
    unsigned long long *x, *y, *z;       // du_dx [S] each
    unsigned long long *q, *sig, *eps;   // du_dp [S] each
    unsigned long long *u, *dl;          // per-slot energy and du_dl [S]
    unsigned long long *pq, *psig, *peps; // du_dp of the scaled-pair part (interpolated), else == q/sig/eps
};

// Accumulator block b (0: contributions shared by all windows, 1 + k: window k)
// lies `block` elements after block 0.
__device__ __forceinline__ Accum acc_block(const Accum &a, size_t block, int b) {
    const size_t o = block * (size_t)b;
    Accum r;
    r.x = a.x + o;
    r.y = a.y + o;
    r.z = a.z + o;
    r.q = a.q + o;
    r.sig = a.sig + o;
    r.eps = a.eps + o;
    r.u = a.u + o;
    r.dl = a.dl + o;
    r.pq = a.pq + o;
    r.psig = a.psig + o;
    r.peps = a.peps + o;
    return r;
}

struct PairArgs {
    int S;
    int row_end;                // slots [0, row_end) act as rows (S, or the interaction group's rows)
    int K;                      // lambda windows
    const float4 *posw;         // [K][S]
    const float4 *prm;          // [K][S]
    const float4 *dprm;         // [K][S]
    const unsigned char *lamdep; // [S]
    const double4 *posw64;      // [K][S] FP64 pair arithmetic (else nullptr)
    const double4 *prm64;       // [K][S]
    const double4 *dprm64;      // [K][S]
    const double *box;
    double beta;
    double cutoff;
    const unsigned *tile_cols;
    const int4 *items;
    // scaled pairs (exclusions / 1-4): original atom indices and scales
    int M;
    const int *pair_idxs;  // [M,2]
    const double *scales;  // [M,2]
    const int *slot_of;    // [N] atom -> slot, nullptr: identity
    int negated;
    Accum acc;             // block 0
    size_t acc_block;      // elements between accumulator blocks
    const int2 *dep_tiles; // [n_dep] (row group, tile) of the lambda-dependent tiles (multi-window)
    DevState *state;
};

__device__ __forceinline__ void red_add(unsigned long long *p, unsigned long long v) { atomicAdd(p, v); }

// The staged slot arrays the pair arithmetic of type Real reads: FP32 float4
// or FP64 double4 copies of the same values.
template <typename Real> struct Staged;
template <> struct Staged<float> {
    using V = float4;
    static __device__ __forceinline__ const float4 *posw(const PairArgs &a) { return a.posw; }
    static __device__ __forceinline__ const float4 *prm(const PairArgs &a) { return a.prm; }
    static __device__ __forceinline__ const float4 *dprm(const PairArgs &a) { return a.dprm; }
    static __device__ __forceinline__ float4 make(float x, float y, float z, float w) { return make_float4(x, y, z, w); }
};
template <> struct Staged<double> {
    using V = double4;
    static __device__ __forceinline__ const double4 *posw(const PairArgs &a) { return a.posw64; }
    static __device__ __forceinline__ const double4 *prm(const PairArgs &a) { return a.prm64; }
    static __device__ __forceinline__ const double4 *dprm(const PairArgs &a) { return a.dprm64; }
    static __device__ __forceinline__ double4 make(double x, double y, double z, double w) {
        return make_double4(x, y, z, w);
    }
};

// ---------------------------------------------------------------------------
// Tile walk: the pairs of a tile (RG rows x 32 columns) that lie within the
// cutoff, and only those.
//
// What bounds it (ncu, forces at 22,840 atoms): no pipe by itself. 64 % of the issue
// slots are taken, 28.6 of 32 lanes per instruction, 65 % of the L1 / shared
// wavefronts, DRAM idle; 34 % of the warps are active and wait longest for loaded
// columns (long_scoreboard, 2.2 cycles per issue). The sweep of every row x column
// that this replaced issued 69.8 M warp instructions there, the walk 43.4 M. Kernel
// times on B200 under ncu, before -> after, bit-identical: forces 92.3 -> 69.2 us,
// all outputs of 12 windows 154 -> 104 (FP64 410 -> 209). CTAs per SM: PAIR_MIN_CTAS;
// loading the next tile's columns ahead costs 2 to 6 %.
//
// Lane l owns column l of the tile: its atom and its sums stay in registers.
// The tile's rows are staged in shared memory once per work item. A tile takes
// two passes: every lane marks the rows within the cutoff of its column (a bit
// mask, distances only, two rows per packed FP32x2 operation), then walks its
// own marked rows, one per step, all lanes with the pair arithmetic at once.
// The list builder puts columns with about as many rows in range next to each
// other, so the lanes of a tile have walks of about the same length (0.80 of
// the lane steps hold a pair; 0.42 of the slots of the tiles do, which is what
// a sweep over all rows x columns spends the pair arithmetic on).
//
// A row's sums are met by several lanes in a step and live in shared memory as
// two 32-bit limbs (bits 0-23 and 24-55 of the fixed-point value): 32-bit
// shared-memory additions are native, 64-bit ones are compare-and-swap loops.
// LIMB_ADDITIONS values up to LIMB_MAX fit the limbs exactly; larger ones (and
// NaN) go to the row's global accumulator as a whole. Lane l starts its walk at
// row l mod RG and each RG-lane group has its own copy of the sums, so the
// lanes of a step mostly meet different words.
// ---------------------------------------------------------------------------
constexpr int LIMB_ADDITIONS = 64;
constexpr long long LIMB_MAX = (1LL << 49) - 1;
static_assert(LIMB_ADDITIONS * 0xffffffLL <= 0xffffffffLL, "low limb");
static_assert(
    LIMB_ADDITIONS * (LIMB_MAX >> 24) <= 0x7fffffffLL && LIMB_ADDITIONS * (-LIMB_MAX >> 24) >= -0x80000000LL, "high limb");

template <typename Real> struct alignas(2 * sizeof(Real)) Vec2 {
    Real a, b;
};

// The rows of one work item, one instance per warp.
template <typename Real, bool DX, bool DP, bool INTERP, int RG> struct alignas(16) WalkRows {
    static constexpr int FIELDS = (DX ? 3 : 0) + (DP ? 3 : 0);
    // tiles between two flushes of the row sums: at most LIMB_ADDITIONS to a word
    static constexpr int FLUSH_TILES = LIMB_ADDITIONS / RG;
    // coordinates row by row for the distance pass, and as pairs for the walk
    Real x[RG], y[RG], z[RG];
    Vec2<Real> xy[RG], zq[RG], se[RG], wd[RG]; // (x, y), (z, q), (sig, eps), (w, dw/dlambda)
    Vec2<Real> dqs[INTERP ? RG : 1];           // (dq/dlambda, dsig/dlambda)
    Real de[INTERP ? RG : 1];                  // deps/dlambda
    Real lo[3], hi[3];                         // smallest and largest row coordinates
    unsigned acc[FIELDS > 0 ? 2 * FIELDS : 1][TILE]; // limbs of the row sums: [field low, high][copy * RG + row]
};

// Sums of the lane's column.
struct ColSums {
    unsigned long long x = 0, y = 0, z = 0, q = 0, sig = 0, eps = 0, u = 0, dl = 0;
};

// What a tile needs besides its atoms, uniform over the launch.
template <typename Real> struct WalkBox {
    Real x, y, z;          // box edges
    Real inv_x, inv_y, inv_z;
    Real cutoff_squared, beta;
};

template <typename Real> __device__ __forceinline__ WalkBox<Real> walk_box(const double *box, double cutoff, double beta) {
    WalkBox<Real> b;
    b.x = box[0];
    b.y = box[4];
    b.z = box[8];
    b.inv_x = 1 / b.x;
    b.inv_y = 1 / b.y;
    b.inv_z = 1 / b.z;
    const Real c = static_cast<Real>(cutoff);
    b.cutoff_squared = c * c;
    b.beta = static_cast<Real>(beta);
    return b;
}

// A value that the limbs hold once it is rounded: |y| < LIMB_MAX rounds to at most
// LIMB_MAX in FP64; in FP32, where LIMB_MAX is 2^49, the next smaller y is an integer.
template <typename Real> __device__ __forceinline__ bool fits_limbs(Real y) { return fabs(y) < static_cast<Real>(LIMB_MAX); }

__device__ __forceinline__ void limbs_add(unsigned (*acc)[TILE], int field, int word, unsigned long long v) {
    atomicAdd(&acc[2 * field][word], static_cast<unsigned>(v) & 0xffffffu);
    atomicAdd(&acc[2 * field + 1][word], static_cast<unsigned>(v >> 24));
}

// Smallest / largest value of the warp; NaNs are passed over. (FP32: one
// instruction in place of ten; forces at 98,000 atoms 242 -> 238 us.)
__device__ __forceinline__ float warp_min(float v) {
    float r;
    asm volatile("redux.sync.min.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}
__device__ __forceinline__ float warp_max(float v) {
    float r;
    asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}
__device__ __forceinline__ double warp_min(double v) {
    for (int o = TILE / 2; o > 0; o >>= 1) {
        v = fmin(v, __shfl_xor_sync(FULL_MASK, v, o));
    }
    return v;
}
__device__ __forceinline__ double warp_max(double v) {
    for (int o = TILE / 2; o > 0; o >>= 1) {
        v = fmax(v, __shfl_xor_sync(FULL_MASK, v, o));
    }
    return v;
}

template <typename Real, bool DX, bool DP, bool INTERP, int RG>
__device__ __forceinline__ void walk_clear(WalkRows<Real, DX, DP, INTERP, RG> &sm, int lane) {
    for (int f = 0; f < 2 * sm.FIELDS; f++) {
        sm.acc[f][lane] = 0;
    }
    __syncwarp();
}

// Stages the rows row_first .. row_first + RG - 1 of one window (slots from
// row_end on: NaN coordinates, which pass no cutoff test). Returns whether any
// row's terms depend on lambda.
template <typename Real, bool DX, bool DP, bool INTERP, int RG>
__device__ __forceinline__ bool walk_load_rows(
    const PairArgs &a, WalkRows<Real, DX, DP, INTERP, RG> &sm, const int lane, const unsigned row_first, const int window) {
    using St = Staged<Real>;
    using V = typename St::V;
    const size_t wo = (size_t)window * a.S;
    const int r = lane & (RG - 1);
    const unsigned i = row_first + r;
    const bool ok = i < (unsigned)a.row_end;
    const Real nan = static_cast<Real>(__int_as_float(0x7fffffff));
    const V pw = ok ? St::posw(a)[wo + i] : St::make(nan, nan, nan, 0);
    const V pr = ok ? St::prm(a)[wo + i] : St::make(0, 0, 0, 0);
    V dp = St::make(0, 0, 0, 0);
    if (INTERP && ok) {
        dp = St::dprm(a)[wo + i];
    }
    // the NaN rows are passed over
    const Real lx = warp_min(pw.x), ly = warp_min(pw.y), lz = warp_min(pw.z);
    const Real hx = warp_max(pw.x), hy = warp_max(pw.y), hz = warp_max(pw.z);
    __syncwarp(); // the previous item's walks are done with the rows
    if (lane < RG) {
        sm.x[r] = pw.x;
        sm.y[r] = pw.y;
        sm.z[r] = pw.z;
        sm.xy[r] = {pw.x, pw.y};
        sm.zq[r] = {pw.z, pr.x};
        sm.se[r] = {pr.y, pr.z};
        sm.wd[r] = {pw.w, pr.w};
        if (INTERP) {
            sm.dqs[r] = {dp.x, dp.y};
            sm.de[r] = dp.z;
        }
    }
    if (lane == 0) {
        sm.lo[0] = lx;
        sm.lo[1] = ly;
        sm.lo[2] = lz;
        sm.hi[0] = hx;
        sm.hi[1] = hy;
        sm.hi[2] = hz;
    }
    __syncwarp();
    return __any_sync(FULL_MASK, pw.w != 0 || (INTERP && (dp.x != 0 || dp.y != 0 || dp.z != 0)));
}

// Adds the rows' sums to the accumulators of the row slots and clears them.
template <typename Real, bool DX, bool DP, bool INTERP, int RG>
__device__ __forceinline__ void walk_flush_rows(
    WalkRows<Real, DX, DP, INTERP, RG> &sm, const int lane, const Accum &out, const unsigned row_first, const int row_end) {
    __syncwarp();
    const unsigned i = row_first + lane;
    const bool writes = lane < RG && i < (unsigned)row_end;
#pragma unroll
    for (int f = 0; f < sm.FIELDS; f++) {
        unsigned long long v = (unsigned long long)sm.acc[2 * f][lane] +
                               ((unsigned long long)(long long)(int)sm.acc[2 * f + 1][lane] << 24);
        sm.acc[2 * f][lane] = 0;
        sm.acc[2 * f + 1][lane] = 0;
#pragma unroll
        for (int o = RG; o < TILE; o <<= 1) {
            v += __shfl_xor_sync(FULL_MASK, v, o);
        }
        if (writes && v != 0) {
            const int k = DX ? f : f + 3;
            unsigned long long *to =
                k == 0 ? out.x : k == 1 ? out.y : k == 2 ? out.z : k == 3 ? out.q : k == 4 ? out.sig : out.eps;
            red_add(to + i, v);
        }
    }
    __syncwarp();
}

// Minimum-image displacement of a coordinate pair: the general form, or the
// image count of the column given as its shift (-box * count).
template <bool WRAP, typename V2>
__device__ __forceinline__ V2 walk_delta2(V2 ci, V2 cj, V2 shift, V2 neg_box, V2 inv_box) {
    if (WRAP) {
        return min_image2(fsub2(ci, cj), neg_box, inv_box);
    }
    return fadd2(fsub2(ci, cj), shift);
}
template <bool WRAP, typename Real>
__device__ __forceinline__ Real walk_delta(Real ci, Real cj, Real shift, Real box, Real inv_box) {
    if (WRAP) {
        return min_image(fsub(ci, cj), box, inv_box);
    }
    return fadd(fsub(ci, cj), shift);
}

// A pair's terms, already scaled to fixed point: the column's to its registers,
// the row's to its limbs, or to its accumulator where the limbs do not hold it.
template <typename Rows, typename Real>
__device__ __forceinline__ void walk_add_force(
    Rows &sm, const int copy, const int r, const unsigned row_first, const Real yx, const Real yy, const Real yz,
    const Accum &out, ColSums &g) {
    const unsigned long long fx = fixed_round(yx);
    const unsigned long long fy = fixed_round(yy);
    const unsigned long long fz = fixed_round(yz);
    g.x -= fx;
    g.y -= fy;
    g.z -= fz;
    if (fits_limbs(yx) && fits_limbs(yy) && fits_limbs(yz)) {
        limbs_add(sm.acc, 0, copy + r, fx);
        limbs_add(sm.acc, 1, copy + r, fy);
        limbs_add(sm.acc, 2, copy + r, fz);
    } else {
        red_add(out.x + row_first + r, fx);
        red_add(out.y + row_first + r, fy);
        red_add(out.z + row_first + r, fz);
        // llrint(-y) equals -llrint(y) except where the conversion
        // saturates (|y| >= 2^63) or y is NaN: add the difference
        if (!fixed_in_range(yx) || !fixed_in_range(yy) || !fixed_in_range(yz)) {
            g.x += fixed_round(-yx) + fx;
            g.y += fixed_round(-yy) + fy;
            g.z += fixed_round(-yz) + fz;
        }
    }
}
template <bool DX, typename Rows, typename Real>
__device__ __forceinline__ void walk_add_charge(
    Rows &sm, const int copy, const int r, const unsigned row_first, const Real y_row, const Real y_col, const Accum &out,
    ColSums &g) {
    const unsigned long long v = fixed_round(y_row);
    g.q += fixed_round(y_col);
    if (fits_limbs(y_row)) {
        limbs_add(sm.acc, DX ? 3 : 0, copy + r, v);
    } else {
        red_add(out.q + row_first + r, v);
    }
}
template <bool DX, typename Rows, typename Real>
__device__ __forceinline__ void walk_add_lj(
    Rows &sm, const int copy, const int r, const unsigned row_first, const Real y_sig, const Real y_eps_row,
    const Real y_eps_col, const Accum &out, ColSums &g) {
    const unsigned long long gs = fixed_round(y_sig), ge = fixed_round(y_eps_row);
    g.sig += gs;
    g.eps += fixed_round(y_eps_col);
    if (fits_limbs(y_sig) && fits_limbs(y_eps_row)) {
        limbs_add(sm.acc, DX ? 4 : 1, copy + r, gs);
        limbs_add(sm.acc, DX ? 5 : 2, copy + r, ge);
    } else {
        red_add(out.sig + row_first + r, gs);
        red_add(out.eps + row_first + r, ge);
    }
}

// The same walk for FP32 pairs without lambda terms, two rows per step: the
// lane's two pairs are the components of packed FP32x2 operations (each
// component rounds as the scalar operation does), which halves the
// arithmetic's instructions and gives each step two independent chains. A lane
// with an odd number of rows computes its last one twice and adds it once.
// Measured on B200 against one row per step, us per call: 98,000 atoms forces
// 252 -> 245, energy 185 -> 169, all outputs 342 -> 321, 12 windows 437 -> 415;
// 22,840 atoms 79.3 -> 77.1, 61.1 -> 57.3, 104.1 -> 99.1, 136.0 -> 131.2; below
// 5,000 atoms no difference. At 5 CTAs/SM (93 registers) 261 / 170 / 339 / 441.
template <bool U, bool DX, bool DP, bool INTERP, bool WRAP, int RG>
__device__ __forceinline__ void walk_two(
    WalkRows<float, DX, DP, INTERP, RG> &sm,
    const int lane,
    const unsigned row_first,
    unsigned m, // rows within the cutoff, rotated right by the lane's first row
    const float4 pwj,
    const float4 prj,
    const float shift_x,
    const float shift_y,
    const float shift_z,
    const WalkBox<float> &b,
    const Accum &out,
    ColSums &g) {
    const int rot = lane & (RG - 1);
    const int copy = lane & ~(RG - 1);
    for (unsigned n = (__reduce_max_sync(FULL_MASK, (unsigned)__popc(m)) + 1) / 2; n > 0; n--) {
        if (m == 0) {
            continue;
        }
        const int ra = (__ffs(m) - 1 + rot) & (RG - 1);
        m &= m - 1;
        const bool two = m != 0;
        const int rb = two ? (__ffs(m) - 1 + rot) & (RG - 1) : ra;
        m &= m - 1;
        const Vec2<float> xya = sm.xy[ra], zqa = sm.zq[ra], xyb = sm.xy[rb], zqb = sm.zq[rb];
        const float2 dx = walk_delta2<WRAP>(make2(xya.a, xyb.a), f2(pwj.x), f2(shift_x), f2(-b.x), f2(b.inv_x));
        const float2 dy = walk_delta2<WRAP>(make2(xya.b, xyb.b), f2(pwj.y), f2(shift_y), f2(-b.y), f2(b.inv_y));
        const float2 dz = walk_delta2<WRAP>(make2(zqa.a, zqb.a), f2(pwj.z), f2(shift_z), f2(-b.z), f2(b.inv_z));
        const float2 d2 = dist2(dx, dy, dz);
        // electrostatics (charge scale 1)
        const float2 inv_d = make2(inv_sqrt(d2.x), inv_sqrt(d2.y));
        const float2 d = fmul2(d2, inv_d);
        const float2 inv_d2 = fmul2(inv_d, inv_d);
        const float2 qi = make2(zqa.b, zqb.b), qj = f2(prj.x);
        const float2 qij_inv = fmul2(fmul2(qi, qj), inv_d);
        float2 erfc_bd;
        const float2 factor = es_factor2(b.beta, d, inv_d2, erfc_bd);
        float2 prefactor = fmul2(qij_inv, factor);
        float2 u = fmul2(qij_inv, erfc_bd);
        if (prj.z != 0) {
            const Vec2<float> sea = sm.se[ra], seb = sm.se[rb];
            const bool lja = sea.b != 0, ljb = seb.b != 0;
            if (lja || ljb) {
                float2 pre_lj = prefactor, u_lj = u, sig_grad, eps_grad;
                lennard_jones2<U>(make2(sea.b, seb.b), f2(prj.z), make2(sea.a, seb.a), f2(prj.y), inv_d, inv_d2, qij_inv,
                                  factor, erfc_bd, u_lj, pre_lj, sig_grad, eps_grad);
                prefactor = make2(lja ? pre_lj.x : prefactor.x, ljb ? pre_lj.y : prefactor.y);
                u = make2(lja ? u_lj.x : u.x, ljb ? u_lj.y : u.y);
                if (DP) {
                    const float2 ys = fmul2(sig_grad, f2(static_cast<float>(FX_EXPONENT_SIG)));
                    const float2 ei =
                        fmul2(fmul2(eps_grad, f2(prj.z)), f2(static_cast<float>(FX_EXPONENT_EPS)));
                    const float2 ej = fmul2(
                        fmul2(eps_grad, make2(sea.b, seb.b)), f2(static_cast<float>(FX_EXPONENT_EPS)));
                    if (lja) {
                        walk_add_lj<DX>(sm, copy, ra, row_first, ys.x, ei.x, ej.x, out, g);
                    }
                    if (two && ljb) {
                        walk_add_lj<DX>(sm, copy, rb, row_first, ys.y, ei.y, ej.y, out, g);
                    }
                }
            }
        }
        const float2 ex = f2(static_cast<float>(FX_EXPONENT));
        if (U) {
            const float2 yu = fmul2(u, ex);
            g.u += fixed_round(yu.x);
            if (two) {
                g.u += fixed_round(yu.y);
            }
        }
        if (DP) {
            const float2 yi = fmul2(fmul2(fmul2(qj, inv_d), erfc_bd), ex);
            const float2 yj = fmul2(fmul2(fmul2(qi, inv_d), erfc_bd), ex);
            walk_add_charge<DX>(sm, copy, ra, row_first, yi.x, yj.x, out, g);
            if (two) {
                walk_add_charge<DX>(sm, copy, rb, row_first, yi.y, yj.y, out, g);
            }
        }
        if constexpr (DX) {
            const float2 yx = fmul2(fmul2(prefactor, dx), ex);
            const float2 yy = fmul2(fmul2(prefactor, dy), ex);
            const float2 yz = fmul2(fmul2(prefactor, dz), ex);
            walk_add_force(sm, copy, ra, row_first, yx.x, yy.x, yz.x, out, g);
            if (two) {
                walk_add_force(sm, copy, rb, row_first, yx.y, yy.y, yz.y, out, g);
            }
        }
    }
}

// One tile, columns j (one per lane; >= S: none), window `window`. Per-pair
// arithmetic and validity follow
// timemachine/cpp/src/kernels/k_nonbonded.cuh:424-546; the column's force is
// the exact negation of the row's (llrint is odd under round-half-even), so it
// is converted once. The energy and du_dl of a pair go to its column.
template <typename Real, bool U, bool DX, bool DL, bool DP, bool INTERP, bool ALCH, bool WRAP, int RG>
__device__ __forceinline__ void walk_pairs(
    WalkRows<Real, DX, DP, INTERP, RG> &sm,
    const int lane,
    const unsigned row_first,
    const unsigned valid_rows, // rows that pair with the lane's column at all
    const typename Staged<Real>::V pwj,
    const typename Staged<Real>::V prj,
    const typename Staged<Real>::V dpj,
    const Real shift_x,
    const Real shift_y,
    const Real shift_z,
    const WalkBox<Real> &b,
    const Accum &out,
    ColSums &g) {
    using V2 = decltype(f2(Real(0)));
    // 1. rows within the cutoff of the lane's column
    unsigned mask = 0;
    {
        const V2 cx = f2(pwj.x), cy = f2(pwj.y), cz = f2(pwj.z);
        const V2 sx = f2(shift_x), sy = f2(shift_y), sz = f2(shift_z);
#pragma unroll
        for (int r = 0; r < RG; r += 2) {
            const Vec2<Real> xr = *reinterpret_cast<const Vec2<Real> *>(&sm.x[r]);
            const Vec2<Real> yr = *reinterpret_cast<const Vec2<Real> *>(&sm.y[r]);
            const Vec2<Real> zr = *reinterpret_cast<const Vec2<Real> *>(&sm.z[r]);
            const V2 dx = walk_delta2<WRAP>(make2(xr.a, xr.b), cx, sx, f2(-b.x), f2(b.inv_x));
            const V2 dy = walk_delta2<WRAP>(make2(yr.a, yr.b), cy, sy, f2(-b.y), f2(b.inv_y));
            const V2 dz = walk_delta2<WRAP>(make2(zr.a, zr.b), cz, sz, f2(-b.z), f2(b.inv_z));
            V2 d2 = dist2(dx, dy, dz);
            if (ALCH) {
                const V2 dw = fsub2(make2(sm.wd[r].a, sm.wd[r + 1].a), f2(pwj.w));
                d2 = madd2(dw, dw, d2, TMNB_DAG_D4);
            }
            if (d2.x < b.cutoff_squared) {
                mask |= 1u << r;
            }
            if (d2.y < b.cutoff_squared) {
                mask |= 2u << r;
            }
        }
        mask &= valid_rows;
    }
    // 2. the lane's rows, from row l mod RG on
    const int rot = lane & (RG - 1);
    const int copy = lane & ~(RG - 1);
    unsigned m = RG == TILE ? __funnelshift_r(mask, mask, rot)
                            : ((mask | (mask << (RG & 31))) >> rot) & (unsigned)((1ull << RG) - 1);
    if constexpr (sizeof(Real) == 4 && !ALCH) {
        walk_two<U, DX, DP, INTERP, WRAP, RG>(
            sm, lane, row_first, m, pwj, prj, shift_x, shift_y, shift_z, b, out, g);
    } else {
        for (unsigned n = __reduce_max_sync(FULL_MASK, (unsigned)__popc(m)); n > 0; n--) {
            if (m == 0) {
                continue;
            }
            const int r = (__ffs(m) - 1 + rot) & (RG - 1);
            m &= m - 1;
            const Vec2<Real> xy = sm.xy[r];
            const Vec2<Real> zq = sm.zq[r];
            const V2 dxy = walk_delta2<WRAP>(
                make2(xy.a, xy.b), make2(pwj.x, pwj.y), make2(shift_x, shift_y), make2(-b.x, -b.y), make2(b.inv_x, b.inv_y));
            const Real delta_x = dxy.x, delta_y = dxy.y;
            const Real delta_z = walk_delta<WRAP>(zq.a, pwj.z, shift_z, b.z, b.inv_z);
            Real d2 = dist2(delta_x, delta_y, delta_z);
            Real delta_w = 0, dw_dl_i = 0;
            if (ALCH) {
                const Vec2<Real> wd = sm.wd[r];
                delta_w = fsub(wd.a, pwj.w);
                dw_dl_i = wd.b;
                d2 = add_w2(d2, delta_w);
            }
            const Real qi = zq.b, qj = prj.x;
            Real u, prefactor, erfc_bd, d, inv_d, inv_d2, qij_inv, factor;
            electrostatics<Real, U>((Real)1, qi, qj, d2, b.beta, d, inv_d, inv_d2, erfc_bd, prefactor, u, qij_inv, factor);
            Real real_du_dl = 0;
            const Real eps_j = prj.z;
            if (eps_j != 0) {
                const Vec2<Real> se = sm.se[r];
                const Real eps_i = se.b;
                if (eps_i != 0) {
                    Real sig_grad, eps_grad;
                    lennard_jones<Real, U>(
                        (Real)1, eps_i, eps_j, se.a, prj.y, inv_d, inv_d2, qij_inv, factor, erfc_bd, u, prefactor, sig_grad,
                        eps_grad);
                    if (DP) {
                        const Real ys = fmul(sig_grad, static_cast<Real>(FX_EXPONENT_SIG));
                        const V2 ye = fmul2(
                            fmul2(f2(eps_grad), make2(eps_j, eps_i)), f2(static_cast<Real>(FX_EXPONENT_EPS)));
                        walk_add_lj<DX>(sm, copy, r, row_first, ys, ye.x, ye.y, out, g);
                    }
                    if (DL && ALCH && INTERP) {
                        real_du_dl = ffma(sig_grad, fadd(sm.dqs[r].b, dpj.y), real_du_dl);
                        real_du_dl = ffma(eps_grad, sum_of_products_rn(eps_j, sm.de[r], eps_i, dpj.z), real_du_dl);
                    }
                }
            }
            if constexpr (DX) {
                const Real ex = static_cast<Real>(FX_EXPONENT);
                const V2 yxy = fmul2(fmul2(f2(prefactor), dxy), f2(ex));
                walk_add_force(sm, copy, r, row_first, yxy.x, yxy.y, fmul(fmul(prefactor, delta_z), ex), out, g);
            }
            if (DP) {
                const V2 yq = fmul2(
                    fmul2(fmul2(make2(qj, qi), f2(inv_d)), f2(erfc_bd)), f2(static_cast<Real>(FX_EXPONENT)));
                walk_add_charge<DX>(sm, copy, r, row_first, yq.x, yq.y, out, g);
            }
            if (DL && ALCH) {
                real_du_dl = ffma(fmul(delta_w, prefactor), fsub(dw_dl_i, prj.w), real_du_dl);
                if (INTERP) {
                    real_du_dl =
                        ffma(fmul(inv_d, erfc_bd), sum_of_products_rn(qj, sm.dqs[r].a, qi, dpj.x), real_du_dl);
                }
                g.dl += to_fixed(real_du_dl, FX_EXPONENT);
            }
            if (U) {
                g.u += to_fixed(u, FX_EXPONENT);
            }
        }
    }
}

// One tile: column j of the lane (>= S: none) against the staged rows; the
// columns' sums go to their accumulators. SHIFT: tiles whose columns have one
// image each take a walk of their own (without it: less code, and the general
// image for every tile).
template <typename Real, bool U, bool DX, bool DL, bool DP, bool INTERP, int RG, bool SHIFT>
__device__ __forceinline__ void walk_tile(
    const PairArgs &a,
    WalkRows<Real, DX, DP, INTERP, RG> &sm,
    const int lane,
    const unsigned row_first,
    const bool rows_alch,
    const unsigned j,
    const int window,
    const WalkBox<Real> &b,
    const Accum &out) {
    using St = Staged<Real>;
    using V = typename St::V;
    const size_t wo = (size_t)window * a.S;
    const bool col_ok = j < (unsigned)a.S;
    const Real nan = static_cast<Real>(__int_as_float(0x7fffffff));
    const V pwj = col_ok ? St::posw(a)[wo + j] : St::make(nan, nan, nan, 0);
    const V prj = col_ok ? St::prm(a)[wo + j] : St::make(0, 0, 0, 0);
    V dpj = St::make(0, 0, 0, 0);
    if (INTERP && col_ok) {
        dpj = St::dprm(a)[wo + j];
    }
    const bool alch = rows_alch || __any_sync(FULL_MASK, pwj.w != 0 || (INTERP && (dpj.x != 0 || dpj.y != 0 || dpj.z != 0)));
    // Image count of the column against the rows. Subtraction, scaling and
    // rounding are monotonic, so where the smallest and the largest row
    // coordinate give the same count, every row between them does, and the
    // column's image is one shift: -box * count (exact for counts up to 2) is
    // what the general form's fused multiply-add adds.
    Real nx = 0, ny = 0, nz = 0;
    bool wrap = true;
    if constexpr (SHIFT) {
        nx = round_half_even(fmul(fsub(sm.lo[0], pwj.x), b.inv_x));
        ny = round_half_even(fmul(fsub(sm.lo[1], pwj.y), b.inv_y));
        nz = round_half_even(fmul(fsub(sm.lo[2], pwj.z), b.inv_z));
        const bool one_image = nx == round_half_even(fmul(fsub(sm.hi[0], pwj.x), b.inv_x)) &&
                               ny == round_half_even(fmul(fsub(sm.hi[1], pwj.y), b.inv_y)) &&
                               nz == round_half_even(fmul(fsub(sm.hi[2], pwj.z), b.inv_z)) && fabs(nx) <= 2 &&
                               fabs(ny) <= 2 && fabs(nz) <= 2;
        wrap = __any_sync(FULL_MASK, col_ok && !one_image);
    }
    // a column of the row group itself pairs with the rows before it
    const unsigned own = j - row_first;
    const unsigned valid = !col_ok ? 0u : (own < (unsigned)RG ? (1u << own) - 1 : FULL_MASK);
    ColSums g;
#define TMB_WALK(ALCH_, WRAP_)                                                                                        \
    walk_pairs<Real, U, DX, DL, DP, INTERP, ALCH_, WRAP_, RG>(                                                        \
        sm, lane, row_first, valid, pwj, prj, dpj, fmul(-b.x, nx), fmul(-b.y, ny), fmul(-b.z, nz), b, out, g)
    if (alch) {
        TMB_WALK(true, true);
    } else if (wrap) {
        TMB_WALK(false, true);
    } else if constexpr (SHIFT) {
        TMB_WALK(false, false);
    }
#undef TMB_WALK
    if (col_ok) {
        if (DX) {
            red_add(out.x + j, g.x);
            red_add(out.y + j, g.y);
            red_add(out.z + j, g.z);
        }
        if (DP) {
            red_add(out.q + j, g.q);
            if (prj.z != 0) {
                red_add(out.sig + j, g.sig);
                red_add(out.eps + j, g.eps);
            }
        }
        if (DL && alch) {
            red_add(out.dl + j, g.dl);
        }
        if (U) {
            red_add(out.u + j, g.u);
        }
    }
}

// One work item: the tiles it.y .. it.y + it.z - 1 of row group it.x. With
// skip_dep, tiles that hold a lambda-dependent atom are left out.
template <typename Real, bool U, bool DX, bool DL, bool DP, bool INTERP, bool SKIP_DEP, int RG, bool SHIFT = true>
__device__ __forceinline__ void walk_item(
    const PairArgs &a,
    WalkRows<Real, DX, DP, INTERP, RG> &sm,
    const int lane,
    const int4 it,
    const int window,
    const WalkBox<Real> &b,
    const Accum &out) {
    const unsigned row_first = (unsigned)(it.x * RG);
    const unsigned i = row_first + (lane & (RG - 1));
    if (SKIP_DEP && __any_sync(FULL_MASK, i < (unsigned)a.row_end && a.lamdep[i])) {
        return; // evaluated per window by the (tile, window) units
    }
    const bool rows_alch = walk_load_rows(a, sm, lane, row_first, window);
    for (int t = 0; t < it.z; t++) {
        const unsigned j = a.tile_cols[((long long)it.y + t) * TILE + lane];
        if (!SKIP_DEP || !__any_sync(FULL_MASK, j < (unsigned)a.S && a.lamdep[j])) {
            walk_tile<Real, U, DX, DL, DP, INTERP, RG, SHIFT>(a, sm, lane, row_first, rows_alch, j, window, b, out);
        }
        // counted over all tiles, so that tiles left out do not put it off
        if ((t + 1) % sm.FLUSH_TILES == 0 && t + 1 < it.z) {
            walk_flush_rows(sm, lane, out, row_first, a.row_end);
        }
    }
    walk_flush_rows(sm, lane, out, row_first, a.row_end);
}

// One scaled pair (exclusion / 1-4 correction), arithmetic of
// timemachine/cpp/src/kernels/k_nonbonded_pair_list.cuh:103-215.
template <typename Real, bool U, bool DX, bool DL, bool DP, bool INTERP>
__device__ __forceinline__ void scaled_pair(
    const PairArgs &a,
    int pair,
    int si,
    int sj,
    int window,
    const Accum &acc_out,
    const Real box_x,
    const Real box_y,
    const Real box_z,
    const Real inv_box_x,
    const Real inv_box_y,
    const Real inv_box_z,
    const Real cutoff_squared) {
    using St = Staged<Real>;
    const size_t wo = (size_t)window * a.S;
    const typename St::V pwi = St::posw(a)[wo + si];
    const typename St::V pwj = St::posw(a)[wo + sj];
    const typename St::V pri = St::prm(a)[wo + si];
    const typename St::V prj = St::prm(a)[wo + sj];
    typename St::V dpi = St::make(0, 0, 0, 0);
    typename St::V dpj = dpi;
    if (INTERP) {
        dpi = St::dprm(a)[wo + si];
        dpj = St::dprm(a)[wo + sj];
    }
    const Real ci_x = pwi.x, ci_y = pwi.y, ci_z = pwi.z, ci_w = pwi.w;
    const Real cj_x = pwj.x, cj_y = pwj.y, cj_z = pwj.z, cj_w = pwj.w;
    const Real qi = pri.x, sig_i = pri.y, eps_i = pri.z, dw_dl_i = pri.w;
    const Real qj = prj.x, sig_j = prj.y, eps_j = prj.z, dw_dl_j = prj.w;
    const Real dq_dl_i = dpi.x, dsig_dl_i = dpi.y, deps_dl_i = dpi.z;
    const Real dq_dl_j = dpj.x, dsig_dl_j = dpj.y, deps_dl_j = dpj.z;
    const Real beta = a.beta;
    const Real charge_scale = a.scales[2 * pair + 0];
    const Real lj_scale = a.scales[2 * pair + 1];

    Real delta_x = fsub(ci_x, cj_x);
    Real delta_y = fsub(ci_y, cj_y);
    Real delta_z = fsub(ci_z, cj_z);
    delta_x = min_image(delta_x, box_x, inv_box_x);
    delta_y = min_image(delta_y, box_y, inv_box_y);
    delta_z = min_image(delta_z, box_z, inv_box_z);
    const Real delta_w = fsub(ci_w, cj_w);
    const Real d2 = add_w2(dist2(delta_x, delta_y, delta_z), delta_w);

    const bool is_vanilla = (ci_w == 0 && dq_dl_i == 0 && dsig_dl_i == 0 && deps_dl_i == 0 && cj_w == 0 &&
                             dq_dl_j == 0 && dsig_dl_j == 0 && deps_dl_j == 0);
    if (!(d2 < cutoff_squared)) {
        return;
    }
    Real u;
    Real erfc_bd;
    Real prefactor;
    Real d;
    Real inv_d;
    Real inv_d2;
    Real qij_inv;
    Real factor;
    electrostatics<Real, true>(
        charge_scale, qi, qj, d2, beta, d, inv_d, inv_d2, erfc_bd, prefactor, u, qij_inv, factor);
    Real real_du_dl = 0;
    unsigned long long g_sig = 0, g_epsi = 0, g_epsj = 0;
    if (eps_i != 0 && eps_j != 0) {
        Real sig_grad;
        Real eps_grad;
        lennard_jones<Real, true>(
            lj_scale, eps_i, eps_j, sig_i, sig_j, inv_d, inv_d2, qij_inv, factor, erfc_bd, u, prefactor, sig_grad,
            eps_grad);
        g_sig = to_fixed(sig_grad, FX_EXPONENT_SIG);
        g_epsi = to_fixed(fmul(eps_grad, eps_j), FX_EXPONENT_EPS);
        g_epsj = to_fixed(fmul(eps_grad, eps_i), FX_EXPONENT_EPS);
        if (INTERP) {
            real_du_dl = ffma(sig_grad, fadd(dsig_dl_i, dsig_dl_j), real_du_dl);
            real_du_dl = ffma(eps_grad, sum_of_products_rn(eps_j, deps_dl_i, eps_i, deps_dl_j), real_du_dl);
        }
    }
    const bool neg = a.negated != 0;
    auto acc = [neg](unsigned long long *p, unsigned long long v) { red_add(p, neg ? (0ULL - v) : v); };
    if (DX) {
        unsigned long long fx, fy, fz, nx, ny, nz;
        to_fixed_pair(fmul(prefactor, delta_x), FX_EXPONENT, fx, nx);
        to_fixed_pair(fmul(prefactor, delta_y), FX_EXPONENT, fy, ny);
        to_fixed_pair(fmul(prefactor, delta_z), FX_EXPONENT, fz, nz);
        acc(acc_out.x + si, fx);
        acc(acc_out.y + si, fy);
        acc(acc_out.z + si, fz);
        acc(acc_out.x + sj, nx);
        acc(acc_out.y + sj, ny);
        acc(acc_out.z + sj, nz);
    }
    if (DP) {
        acc(acc_out.pq + si, to_fixed(fmul(fmul(fmul(charge_scale, qj), inv_d), erfc_bd), FX_EXPONENT));
        acc(acc_out.pq + sj, to_fixed(fmul(fmul(fmul(charge_scale, qi), inv_d), erfc_bd), FX_EXPONENT));
        acc(acc_out.psig + si, g_sig);
        acc(acc_out.peps + si, g_epsi);
        acc(acc_out.psig + sj, g_sig);
        acc(acc_out.peps + sj, g_epsj);
    }
    if (DL && !is_vanilla) {
        real_du_dl = ffma(fmul(delta_w, prefactor), fsub(dw_dl_i, dw_dl_j), real_du_dl);
        if (INTERP) {
            real_du_dl = ffma(
                fmul(fmul(charge_scale, inv_d), erfc_bd), sum_of_products_rn(qj, dq_dl_i, qi, dq_dl_j), real_du_dl);
        }
        acc(acc_out.dl + si, to_fixed(real_du_dl, FX_EXPONENT));
    }
    if (U) {
        acc(acc_out.u + si, to_fixed(u, FX_EXPONENT));
    }
}

// Multi-window calls: lists the tiles with at least one lambda-dependent row
// or column atom (the tiles the pair kernel evaluates once per window). One
// warp per work item, grid-stride.
struct DepArgs {
    int S;
    int rows; // slots per row group
    int row_end;
    const int4 *items;
    const unsigned *tile_cols;
    const unsigned char *lamdep;
    int2 *dep_tiles;
};

// The list only changes with the tile list or the atoms' lambda dependence,
// so a call with neither keeps the previous one (state->dep_dirty).
static __global__ void k_dep_tiles(DepArgs a, DevState *state) {
    grid_dependency_wait();
    if (state->error || !state->dep_dirty) {
        return;
    }
    const int lane = threadIdx.x & 31;
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int n_warps = (gridDim.x * blockDim.x) >> 5;
    const unsigned S = (unsigned)a.S;
    const int n_items = state->n_items;
    for (int w = warp; w < n_items; w += n_warps) {
        const int4 it = a.items[w];
        const unsigned i = (unsigned)(it.x * a.rows + (lane & (a.rows - 1)));
        const bool row_dep = i < (unsigned)a.row_end && a.lamdep[i];
        for (int t = 0; t < it.z; t++) {
            const int tile = it.y + t;
            const unsigned j = a.tile_cols[(long long)tile * TILE + lane];
            if (__any_sync(FULL_MASK, row_dep || (j < S && a.lamdep[j])) && lane == 0) {
                a.dep_tiles[atomicAdd(&state->n_dep, 1)] = make_int2(it.x, tile);
            }
        }
    }
}

// The warp's next work unit: n_first + the counter's value.
__device__ __forceinline__ int next_unit(int *counter, int n_first, int lane) {
    int v = 0;
    if (lane == 0) {
        v = atomicAdd(counter, 1);
    }
    return n_first + __shfl_sync(FULL_MASK, v, 0);
}

// CTAs per SM the compiler must fit the pair kernel to (its register budget). FP32 on
// B200, us per call at 5 / 6 / 7 / 8, 22,840 and 98,000 atoms: forces 75.1 / 71.2 / 69.7 /
// 68.8 and 256 / 239 / 231 / 225, all outputs 96.7 / 93.1 / 96.2 / 103.7 and 331 / 314 /
// 322 / 347, 12 windows 117 / 112 / 117 / 126 and 416 / 392 / 407 / 437.
template <typename Real> constexpr int PAIR_MIN_CTAS = sizeof(Real) == 4 ? 6 : 5;

// Persistent pair kernel over dynamically scheduled work units:
//   [0, n_items)                 tile work items (row group, first tile, count);
//   MULTI only: [n_items, + n_dep*K)  one lambda-dependent tile at one window;
//   then                         chunks of 32 scaled pairs (one per lane).
// MULTI (K > 1 windows): the tile items skip lambda-dependent tiles and add
// into the shared accumulator block; each (tile, window) unit adds into the
// window's block; a lambda-dependent scaled pair is evaluated for every window.
template <typename Real, bool U, bool DX, bool DL, bool DP, bool INTERP, bool MULTI, int RG = TILE>
__global__ void __launch_bounds__(128, PAIR_MIN_CTAS<Real>) k_pair(PairArgs a) {
    __shared__ WalkRows<Real, DX, DP, INTERP, RG> rows[4];
    grid_dependency_wait();
    if (a.state->error) {
        return;
    }
    const int lane = threadIdx.x & 31;
    WalkRows<Real, DX, DP, INTERP, RG> &sm = rows[threadIdx.x >> 5];
    walk_clear(sm, lane);
    const WalkBox<Real> b = walk_box<Real>(a.box, a.cutoff, a.beta);
    const int n_items = a.state->n_items;
    const int n_dep_units = MULTI ? a.state->n_dep * a.K : 0;
    if (MULTI && blockIdx.x == 0 && threadIdx.x == 0 && !a.state->error) {
        // k_dep_tiles (before this launch) has redone the list; after an
        // error it did not, so the list stays dirty for the next call
        a.state->dep_dirty = 0;
    }
    const int n_tiles_units = n_items + n_dep_units;
    const int n_total = n_tiles_units + (a.M + TILE - 1) / TILE;

    // the first unit of a warp is its own number, the others come from the
    // counter: thousands of warps asking for their first one at once (and, in
    // a small system, for a second one that does not exist) wait for one another
    const int n_warps = gridDim.x * (blockDim.x / TILE);
    for (int item = (blockIdx.x * blockDim.x + threadIdx.x) / TILE; item < n_total;
         item = next_unit(&a.state->next_item, n_warps, lane)) {
        if (item >= n_tiles_units) {
            const int pair = (item - n_tiles_units) * TILE + lane;
            if (pair < a.M) {
                const int atom_i = a.pair_idxs[2 * pair + 0];
                const int atom_j = a.pair_idxs[2 * pair + 1];
                const int si = a.slot_of ? a.slot_of[atom_i] : atom_i;
                const int sj = a.slot_of ? a.slot_of[atom_j] : atom_j;
                const bool dep = MULTI && (a.lamdep[si] || a.lamdep[sj]);
                for (int k = 0; k < (dep ? a.K : 1); k++) {
                    scaled_pair<Real, U, DX, DL, DP, INTERP>(
                        a, pair, si, sj, k, acc_block(a.acc, a.acc_block, dep ? 1 + k : 0), b.x, b.y, b.z, b.inv_x,
                        b.inv_y, b.inv_z, b.cutoff_squared);
                }
            }
            continue;
        }
        int4 it;
        int window = 0;
        if (MULTI && item >= n_items) {
            const int unit = item - n_items;
            const int2 dt = a.dep_tiles[unit / a.K];
            window = unit % a.K;
            it = make_int4(dt.x, dt.y, 1, 0);
            walk_item<Real, U, DX, DL, DP, INTERP, false, RG>(
                a, sm, lane, it, window, b, acc_block(a.acc, a.acc_block, 1 + window));
            continue;
        }
        it = a.items[item];
        walk_item<Real, U, DX, DL, DP, INTERP, MULTI, RG>(a, sm, lane, it, 0, b, a.acc);
    }
}

// ---------------------------------------------------------------------------
// Scatter of the slot-ordered accumulators into the caller's outputs (which
// accumulate, +=). Window k's result is the
// shared block plus block 1 + k (one window: block 0 only).
// du_dp of interpolated potentials is split into the lambda=0 and lambda=1
// halves per potential part, with the rounding of
// timemachine/cpp/src/kernels/k_lambda_transformer_jit.cuh:100-137.
// ---------------------------------------------------------------------------
struct FinalizeArgs {
    int N;
    int S;
    int K;
    double f_dp[MAX_WINDOWS][3]; // interpolated: f(lambda_k) of the charge, sigma and epsilon transforms
    const int *set_atoms; // [S] atoms of the evaluated set in ascending order, nullptr: 0..S-1
    const int *slot_of;   // [N] atom -> slot, nullptr: identity
    int take;             // 1: zero each accumulator after reading it; 0: the caller zeroes them
    Accum acc;
    size_t acc_block;
    int split_pair_dp; // 1: acc.pq/psig/peps are separate buffers
    int interpolated;
    unsigned long long *du_dx; // [K][N,3] (window stride out_stride_x)
    unsigned long long *du_dp; // [K][P]
    unsigned long long *du_dl; // [K][N]
    unsigned long long *u;     // [K][N]
    size_t stride_x, stride_p, stride_n;
    const DevState *state;
};

__device__ __forceinline__ unsigned long long interp_part(double f, unsigned long long v, unsigned long long e) {
    const double real = static_cast<double>(static_cast<long long>(v)) / e;
    return static_cast<unsigned long long>(llrint((f * real) * e));
}

__device__ __forceinline__ unsigned long long take(unsigned long long *p) {
    const unsigned long long v = *p;
    *p = 0;
    return v;
}

// One thread per (window k, set atom), consecutive threads on consecutive
// atoms, so the output updates are coalesced and the slot-ordered
// accumulators are gathered through slot_of. Only the accumulators of
// requested outputs are read (the others are not cleared and may hold an
// earlier call's sums). take = 1 zeroes each accumulator after the read (one
// window: every slot is read by exactly one thread). Outputs are added with integer atomics, so other
// potentials may accumulate into the same buffers concurrently (the sums are
// order-independent).
static __global__ void k_finalize(FinalizeArgs a) {
    grid_dependency_wait();
    const bool ok = a.state->error == 0;
    const bool multi = a.K > 1;
    const size_t total = (size_t)a.S * (size_t)a.K;
    const Accum &c = a.acc;
    for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < total; t += (size_t)gridDim.x * blockDim.x) {
        const int k = (int)(t / (size_t)a.S);
        const int idx = (int)(t - (size_t)k * a.S);
        const int atom = a.set_atoms ? a.set_atoms[idx] : idx;
        const int s = a.slot_of ? a.slot_of[atom] : atom;
        const size_t o = a.acc_block * (size_t)(1 + k) + s;
        auto get = [&](unsigned long long *p) -> unsigned long long {
            if (multi) {
                return p[s] + p[o];
            }
            return a.take ? take(p + s) : p[s];
        };
        if (a.du_dx) {
            const unsigned long long vx = get(c.x), vy = get(c.y), vz = get(c.z);
            if (ok) {
                unsigned long long *out = a.du_dx + a.stride_x * k + 3 * (size_t)atom;
                atomicAdd(out + 0, vx);
                atomicAdd(out + 1, vy);
                atomicAdd(out + 2, vz);
            }
        }
        if (a.du_dp) {
            unsigned long long v0[3] = {get(c.q), get(c.sig), get(c.eps)};
            unsigned long long v1[3] = {0, 0, 0};
            if (a.split_pair_dp) {
                v1[0] = get(c.pq);
                v1[1] = get(c.psig);
                v1[2] = get(c.peps);
            }
            if (ok) {
                const unsigned long long ex[3] = {FX_EXPONENT, FX_EXPONENT_SIG, FX_EXPONENT_EPS};
                unsigned long long *out = a.du_dp + a.stride_p * k;
                for (int d = 0; d < 3; d++) {
                    if (a.interpolated) {
                        const double f = a.f_dp[k][d];
                        unsigned long long lo = interp_part(1 - f, v0[d], ex[d]) + interp_part(1 - f, v1[d], ex[d]);
                        unsigned long long hi = interp_part(f, v0[d], ex[d]) + interp_part(f, v1[d], ex[d]);
                        atomicAdd(out + 3 * (size_t)atom + d, lo);
                        atomicAdd(out + 3 * ((size_t)a.N + atom) + d, hi);
                    } else {
                        atomicAdd(out + 3 * (size_t)atom + d, v0[d] + v1[d]);
                    }
                }
            }
        }
        if (a.u) {
            const unsigned long long vu = get(c.u);
            if (ok) {
                atomicAdd(a.u + a.stride_n * k + atom, vu);
            }
        }
        if (a.du_dl) {
            const unsigned long long vl = get(c.dl);
            if (ok) {
                atomicAdd(a.du_dl + a.stride_n * k + atom, vl);
            }
        }
    }
}

} // namespace tmb
