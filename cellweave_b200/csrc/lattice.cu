// CPM lattice: CpmLattice of crates/engine/src/cpm.rs on the device.
//
// The reference's Monte Carlo step is sequential: N attempts at random
// pixels, each seeing every flip before it (cpm.rs:734-772).  Here one step
// is a sequence of sublattice passes.  Pixels are coloured so that no pixel
// of a colour lies within the contact reach of another (the chessboard for
// contact across faces; a period R+1 in every axis for a reach of Chebyshev
// radius R); a pass makes one copy attempt at every pixel of one colour.
// Attempts of one pass never read a pixel another of them writes; they meet
// only through the volume and surface records of cells they share.  A pass
// runs its attempts as the sequence in a per-pass priority order would (each
// seeing the records every earlier one left): attempts that share no cell run
// at once, those that share one in priority order, each handing the cell's
// records to the next, or in rounds (k_cpm_sweep).  So a pass is
// deterministic whatever the thread schedule, and keeps the sequential
// sweep's volume statistics.  The colours are swept in an order shuffled anew
// every step.
//
// Each attempt is the reference's try_flip (cpm.rs:797-838): a neighbour
// across a face drawn uniformly, no proposal from or into an obstacle or
// within one cell, Delta-H = contact (cpm.rs:851-876) + volume
// (cpm.rs:879-894) [+ surface, an extension], accepted when Delta-H <= 0 or
// u < exp(-Delta-H / T).  Draws come from Philox4x32-10 keyed by the
// history's seed, counter (pixel, step, 0, 0).  This file is built without
// fused multiply-add so that Delta-H rounds as the reference's does.
#include <algorithm>
#include <array>
#include <cmath>
#include <cstring>

#include "cw_internal.cuh"

using namespace cw;

namespace {

constexpr int T = 256;
constexpr int32_t OBST = -1;

struct LatView {
    int32_t *grid;
    const int32_t *type;
    int32_t *volume;
    const int32_t *vsnap;
    const int32_t *target;
    const double *lambda;
    int32_t *surface;
    const int32_t *ssnap;
    const int32_t *tsurf;
    const double *lsurf;
    const int4 *dims;
    const int64_t *off;
    const int64_t *cell_off;
    const uint2 *keys;
    int32_t K;
    int32_t nreach;
    int32_t period;
    int32_t ncol;
    double across;
    double temperature;
    int32_t surface_on;
    int32_t copy_moore;
    uint32_t take_below;   // sub-sweeps: a pixel attempts when its draw is below this (0: every pixel)
    const int32_t *span;   // volumes: the pixels a Monte Carlo step visits (x0 y0 z0 x1 y1 z1 a history)
};

struct Tables {
    double J[64];
    int8_t reach[3 * 124];
};

__device__ __forceinline__ int32_t kind_of(const int32_t *type_h, int64_t cap, int32_t id) {
    if (id < 0 || id >= cap) return 0;  // the obstacle reads as the medium (cpm.rs:908-917)
    return __ldg(type_h + id);
}

// von_neumann, cpm.rs:922-944: y-1, y+1, x-1, x+1, z-1, z+1, clipped; as a
// mask of the six directions in that order (bit k: direction k exists), so
// that the neighbours live in registers.
struct Vn {
    unsigned mask;
    int64_t w, slice;
    __device__ __forceinline__ int count() const { return __popc(mask); }
    __device__ __forceinline__ bool has(int k) const { return (mask >> k) & 1u; }
    __device__ __forceinline__ int64_t step(int k) const {
        return k == 0 ? -w : k == 1 ? w : k == 2 ? -1 : k == 3 ? 1 : k == 4 ? -slice : slice;
    }
    // the offset of the j-th existing neighbour (j < count)
    __device__ __forceinline__ int64_t nth(int j) const { return step(__fns(mask, 0, j + 1)); }
};
// The copy neighbourhood with Moore copies: every in-box pixel at Chebyshev
// distance 1, bit k = (dz + 1) 9 + (dy + 1) 3 + (dx + 1) (the centre, 13, never
// set), taken in that order (the oracle's or_copy_neighbours).
struct Moore {
    unsigned mask;
    int64_t w, slice;
    __device__ __forceinline__ int count() const { return __popc(mask); }
    __device__ __forceinline__ int64_t step(int k) const {
        return (int64_t)(k / 9 - 1) * slice + (int64_t)((k / 3) % 3 - 1) * w + (k % 3 - 1);
    }
    __device__ __forceinline__ int64_t nth(int j) const { return step(__fns(mask, 0, j + 1)); }
};
__device__ __forceinline__ Moore moore_of(int4 dm, int x, int y, int z) {
    Moore m;
    m.w = dm.x;
    m.slice = (int64_t)dm.x * dm.y;
    m.mask = 0u;
    const int deep = dm.z > 1 ? 1 : 0;
    for (int dz = -deep; dz <= deep; ++dz)
        for (int dy = -1; dy <= 1; ++dy)
            for (int dx = -1; dx <= 1; ++dx) {
                if ((dx | dy | dz) == 0) continue;
                if (x + dx < 0 || x + dx >= dm.x || y + dy < 0 || y + dy >= dm.y || z + dz < 0 || z + dz >= dm.z)
                    continue;
                m.mask |= 1u << ((dz + 1) * 9 + (dy + 1) * 3 + (dx + 1));
            }
    return m;
}

__device__ __forceinline__ Vn vn_of(int4 dm, int x, int y, int z) {
    Vn v;
    v.w = dm.x;
    v.slice = (int64_t)dm.x * dm.y;
    v.mask = (y > 0 ? 1u : 0u) | (y + 1 < dm.y ? 2u : 0u) | (x > 0 ? 4u : 0u) | (x + 1 < dm.x ? 8u : 0u) |
             (z > 0 ? 16u : 0u) | (z + 1 < dm.z ? 32u : 0u);
    return v;
}

// contact_delta_h (cpm.rs:851-876) on history grid `g`; *num before the division.
__device__ __forceinline__ double contact_delta(const int32_t *g, int4 dm, int x, int y, int z, int32_t src,
                                int32_t dst, const int32_t *type_h, int64_t cap, const double *sJ, int K,
                                const int8_t *reach, int nreach, double across, int64_t i, Vn vn, double *num) {
    int32_t ks = kind_of(type_h, cap, src), kd = kind_of(type_h, cap, dst);
    double dh = 0.0;
    if (nreach > 0) {
        // a batch of neighbours' ids, then their kinds, in flight at once (one at
        // a time each waits for two reads); added in the reach's order
        constexpr int NB = 13;
        for (int k0 = 0; k0 < nreach; k0 += NB) {
            int32_t nb[NB], kn[NB];
            unsigned in = 0;
#pragma unroll
            for (int q = 0; q < NB; ++q) {
                const int k = k0 + q;
                nb[q] = 0;
                if (k >= nreach) continue;
                const int a = x + reach[3 * k], b = y + reach[3 * k + 1], c = z + reach[3 * k + 2];
                if (a < 0 || b < 0 || c < 0 || a >= dm.x || b >= dm.y || c >= dm.z) continue;
                in |= 1u << q;
                nb[q] = g[((int64_t)c * dm.y + b) * dm.x + a];
            }
#pragma unroll
            for (int q = 0; q < NB; ++q) kn[q] = kind_of(type_h, cap, nb[q]);
#pragma unroll
            for (int q = 0; q < NB; ++q) {
                if (!((in >> q) & 1u)) continue;
                const double ed = dst == nb[q] ? 0.0 : sJ[kd * K + kn[q]];
                const double es = src == nb[q] ? 0.0 : sJ[ks * K + kn[q]];
                dh += ed - es;
            }
        }
        *num = dh;
        return dh / across;
    }
#pragma unroll
    for (int k = 0; k < 6; ++k) {
        if (!vn.has(k)) continue;
        int32_t nb = g[i + vn.step(k)];
        int32_t kn = kind_of(type_h, cap, nb);
        double ed = dst == nb ? 0.0 : sJ[kd * K + kn];
        double es = src == nb ? 0.0 : sJ[ks * K + kn];
        dh += ed - es;
    }
    *num = dh;
    return dh;
}

// volume_delta_h, cpm.rs:879-894: each cell's change of lambda (V - V_target)^2
// on losing (source) or gaining (copied) a pixel, added in that order.
__device__ __forceinline__ double volume_terms(bool has_src, int32_t vs, int32_t ts, double ls, bool has_dst, int32_t vd,
                                               int32_t td, double ld) {
    double dh = 0.0;
    if (has_src) {
        const double v = (double)vs, vt = (double)ts;
        const double a = v - 1.0 - vt, b = v - vt;
        dh += ls * (a * a - b * b);
    }
    if (has_dst) {
        const double v = (double)vd, vt = (double)td;
        const double a = v + 1.0 - vt, b = v - vt;
        dh += ld * (a * a - b * b);
    }
    return dh;
}
// The same on the volumes given (c0: the history's first cell).
__device__ __forceinline__ double volume_delta(const int32_t *vol, const int32_t *target, const double *lambda,
                                               int64_t c0, int32_t src, int32_t dst) {
    int32_t vs = 0, ts = 0, vd = 0, td = 0;
    double ls = 0.0, ld = 0.0;
    if (src != 0) { vs = vol[c0 + src]; ts = target[c0 + src]; ls = lambda[c0 + src]; }
    if (dst != 0) { vd = vol[c0 + dst]; td = target[c0 + dst]; ld = lambda[c0 + dst]; }
    return volume_terms(src != 0, vs, ts, ls, dst != 0, vd, td, ld);
}

__device__ __forceinline__ void surface_change(const int32_t *g, int64_t i, Vn vn, int32_t src, int32_t dst,
                                               int32_t &dsrc, int32_t &ddst) {
    int eq_s = 0, eq_d = 0;
#pragma unroll
    for (int k = 0; k < 6; ++k) {
        if (!vn.has(k)) continue;
        int32_t nb = g[i + vn.step(k)];
        eq_s += nb == src;
        eq_d += nb == dst;
    }
    const int nvn = vn.count();
    dsrc = eq_s - (nvn - eq_s);
    ddst = (nvn - eq_d) - eq_d;
}

__device__ __forceinline__ double surface_terms(bool has_src, int32_t ss, int32_t tss, double lss, int32_t dsrc,
                                                bool has_dst, int32_t sd, int32_t tsd, double lsd, int32_t ddst) {
    double dh = 0.0;
    if (has_src) {
        const double s = (double)ss, st = (double)tss;
        const double a = s + (double)dsrc - st, b = s - st;
        dh += lss * (a * a - b * b);
    }
    if (has_dst) {
        const double s = (double)sd, st = (double)tsd;
        const double a = s + (double)ddst - st, b = s - st;
        dh += lsd * (a * a - b * b);
    }
    return dh;
}
__device__ __forceinline__ double surface_delta(const int32_t *surf, const int32_t *tsurf, const double *lsurf,
                                                int64_t c0, int32_t src, int32_t dst, int32_t dsrc, int32_t ddst) {
    int32_t ss = 0, tss = 0, sd = 0, tsd = 0;
    double lss = 0.0, lsd = 0.0;
    if (src > 0) { ss = surf[c0 + src]; tss = tsurf[c0 + src]; lss = lsurf[c0 + src]; }
    if (dst > 0) { sd = surf[c0 + dst]; tsd = tsurf[c0 + dst]; lsd = lsurf[c0 + dst]; }
    return surface_terms(src > 0, ss, tss, lss, dsrc, dst > 0, sd, tsd, lsd, ddst);
}

// The colour order of the current step for every history: a Fisher-Yates
// shuffle driven by Philox(all-ones, step, 1, i); with `pass_keys`, each
// pass's priority key, word 0 of Philox(all-ones - 1, step, 2, colour);
// advances the step counter, and clears the sweep's barrier words and counts
// (the eight 32-bit words at `words`).
__global__ void k_colour_order(const uint2 *keys, int nh, int ncol, uint32_t *mcs_ctr, uint32_t *mcs_cur,
                               int32_t *perm, uint32_t *pass_keys, uint32_t *words) {
    // one block: every thread reads the counter before thread 0 advances it
    uint32_t m = *mcs_ctr;
    if (threadIdx.x < 8) words[threadIdx.x] = 0u;
    for (int h = threadIdx.x; h < nh; h += blockDim.x) {
        int32_t p[27];
        for (int i = 0; i < ncol; ++i) p[i] = i;
        uint2 k = keys[h];
        for (int i = ncol - 1; i > 0; --i) {
            uint4 r = philox(0xFFFFFFFFu, m, 1u, (uint32_t)i, k.x, k.y);
            int j = (int)(((uint64_t)r.x * (uint64_t)(i + 1)) >> 32);
            int32_t t = p[i]; p[i] = p[j]; p[j] = t;
        }
        for (int i = 0; i < ncol; ++i) perm[h * ncol + i] = p[i];
        if (pass_keys)
            for (int i = 0; i < ncol; ++i)
                pass_keys[h * ncol + i] = philox(0xFFFFFFFEu, m, 2u, (uint32_t)p[i], k.x, k.y).x;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        *mcs_cur = m;
        *mcs_ctr = m + 1;
    }
}

// The rows (y, z) that hold pixels of a colour inside the box b = (x0, y0, z0,
// x1, y1, z1) (inclusive) of a history, `rows` of them (none in an empty box).
// Colour classes: the chessboard (x + y + z) mod 2 for period 0, else the
// residues of x, y, z modulo the period.  (32-bit index arithmetic: a
// history holds fewer than 2^31 pixels.)
struct ColourRows {
    uint32_t rows, ny;  // rows, and how many of them a slice has
    int f[3], step;     // the first pixel along each axis (chessboard: of the box) and the spacing
    int last, nx0;      // the box's last x; a row's count of the colour (chessboard: its colour)
    bool board;
    __device__ __forceinline__ ColourRows(const int (&b)[6], int period, int colour) {
        board = period == 0;
        step = board ? 2 : period;
        last = b[3];
        nx0 = colour;
        uint32_t n[3];
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            f[a] = b[a];
            n[a] = b[a] <= b[3 + a] ? (uint32_t)(b[3 + a] - b[a] + 1) : 0u;
        }
        if (!board) {
            const int c[3] = {colour % period, (colour / period) % period, colour / (period * period)};
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                f[a] = b[a] + ((c[a] - b[a] % period + period) % period);
                n[a] = f[a] <= b[3 + a] ? (uint32_t)((b[3 + a] - f[a]) / period + 1) : 0u;
            }
            nx0 = (int)n[0];
        }
        ny = n[1];
        rows = n[0] ? n[1] * n[2] : 0u;
    }
    // row `row` (below `rows`): its y and z, its first pixel of the colour and their count
    __device__ __forceinline__ void at(uint32_t row, int &y, int &z, int &fx, int &nx) const {
        const uint32_t q = rows == ny ? 0u : row / ny;
        y = (int)(row - q * ny);
        z = (int)q;
        if (board) {
            y += f[1];
            z += f[2];
            fx = f[0] + ((nx0 - f[0] - y - z) & 1);
            nx = fx <= last ? (last - fx) / 2 + 1 : 0;
        } else {
            y = f[1] + step * y;
            z = f[2] + step * z;
            fx = f[0];
            nx = nx0;
        }
    }
};

// How the pixels of one colour in a box of side wx are dealt to items of 32 `useg`
// of them: a row's pixels (`n` at most) in `segs` items of their own, or, where
// that would leave more than an eighth of the lanes without a pixel, the rows one
// behind another (a division a pixel).  4,096 histories of 64 x 64, a Monte Carlo
// step, rows in segments of 128 and the histories' plan walked one at a time ->
// this and 32 histories a step: 3.36 -> 2.10 ms (order 3: 6.30 -> 3.08), and a
// quarter of the scratch.
struct ColourItems {
    uint32_t n, segs;
    bool packed;
    __host__ __device__ __forceinline__ ColourItems(uint32_t wx, int period, int useg) {
        n = period == 0 ? (wx + 1) / 2 : (wx + period - 1) / period;  // (a side is below 2^16)
        segs = (n + 32 * useg - 1) / (32 * useg);
        packed = segs * 32 * useg * 8 > n * 9;
    }
};
// A box's items.
__host__ __device__ __forceinline__ int64_t colour_items(int64_t wx, int64_t wy, int64_t wz, int period, int useg) {
    if (wx <= 0 || wy <= 0 || wz <= 0) return 0;
    const int64_t rows = period == 0 ? wy * wz : ((wy + period - 1) / period) * ((wz + period - 1) / period);
    const ColourItems it((uint32_t)wx, period, useg);
    return it.packed ? (rows * it.n + 32 * useg - 1) / (32 * useg) : rows * it.segs;
}

// MurmurHash3's 32-bit finaliser (Appleby): a bijection of 32-bit words, so
// the pixels of one history get distinct priorities in a pass.
__device__ __forceinline__ uint32_t fmix32(uint32_t h) {
    h ^= h >> 16;
    h *= 0x85ebca6bu;
    h ^= h >> 13;
    h *= 0xc2b2ae35u;
    h ^= h >> 16;
    return h;
}

constexpr uint32_t NONE = 0xFFFFFFFFu;

// One copy attempt of a pass, with everything about it that the pass cannot
// change: the pixels of a colour lie outside one another's reach, so the
// contact term, the surface counts' changes and the draws are fixed when the
// pass starts; only the volume and surface records move.  One line of memory.
struct __align__(128) Attempt {
    double contact;            // contact Delta-H (cpm.rs:851-876)
    double limit;              // Delta-H below it is accepted, above it rejected (decide)
    double ls, ld;             // lambda of the source and of the copied cell
    int32_t ts, td;            // their target volumes
    uint32_t cs, cd;           // their records (NONE: the medium)
    uint32_t next_s, next_d;   // the attempt after this one on each (link; NONE: the last)
    int32_t dst;               // the copied id
    int32_t dsurf;             // surface changes of source and copied cell (int16 each)
    int64_t gi;                // the pixel in the batch's flat order
    uint32_t u0, u1;           // the acceptance draw's words
    double lss, lsd;           // with a surface constraint: the surface lambdas
    int32_t tss, tsd;          // and target surfaces
    uint32_t prio;             // the pass priority
    int32_t src;               // the source id
    uint2 where;               // history | z << 16, x | y << 16
    uint32_t pad[2];
};
static_assert(sizeof(Attempt) == 128, "an attempt is one line");

// The same for a sweep that runs every pass by rounds in little memory: what the
// cells' records hold is read there.
struct __align__(16) LeanAttempt {
    uint32_t cs, cd, prio;
    int32_t dst;
    int64_t gi;
    uint32_t u0, u1;
    union {
        double contact;
        uint2 where;  // until the contact is taken
    };
    int32_t dsurf, src;
};
static_assert(sizeof(LeanAttempt) == 48, "a lean attempt is three 16-byte words");

// What running an attempt takes, read by words of 16 bytes (a copy of the
// struct goes through local memory).
struct Terms {
    double contact, limit, ls, ld, lss, lsd;
    int64_t gi;
    int32_t ts, td, tss, tsd, dst, dsurf;
    uint32_t cs, cd, next_s, next_d, u0, u1;
    __device__ __forceinline__ void read(const Attempt *a, bool surface) {
        const double2 *d = (const double2 *)a;
        const int4 *w = (const int4 *)a;
        const double2 d0 = d[0], d1 = d[1];
        const int4 w2 = w[2], w3 = w[3], w4 = w[4];
        contact = d0.x;
        limit = d0.y;
        ls = d1.x;
        ld = d1.y;
        ts = w2.x;
        td = w2.y;
        cs = (uint32_t)w2.z;
        cd = (uint32_t)w2.w;
        next_s = (uint32_t)w3.x;
        next_d = (uint32_t)w3.y;
        dst = w3.z;
        dsurf = w3.w;
        gi = (int64_t)(((uint64_t)(uint32_t)w4.y << 32) | (uint32_t)w4.x);
        u0 = (uint32_t)w4.z;
        u1 = (uint32_t)w4.w;
        lss = lsd = 0.0;
        tss = tsd = 0;
        if (surface) {
            const double2 d5 = d[5];
            const int4 w6 = w[6];
            lss = d5.x;
            lsd = d5.y;
            tss = w6.x;
            tsd = w6.y;
        }
    }
    __device__ __forceinline__ void read(const LeanAttempt *a, const LatView &L, bool surface) {
        const int4 w0 = ((const int4 *)a)[0], w1 = ((const int4 *)a)[1];
        cs = (uint32_t)w0.x;
        cd = (uint32_t)w0.y;
        dst = w0.w;
        gi = (int64_t)(((uint64_t)(uint32_t)w1.y << 32) | (uint32_t)w1.x);
        u0 = (uint32_t)w1.z;
        u1 = (uint32_t)w1.w;
        contact = a->contact;
        dsurf = a->dsurf;
        limit = (double)NAN;  // (the exponential is taken)
        ls = ld = lss = lsd = 0.0;
        ts = td = tss = tsd = 0;
        next_s = next_d = NONE;
        if (cs != NONE) {
            ts = __ldg(L.target + cs);
            ls = __ldg(L.lambda + cs);
            if (surface) { tss = __ldg(L.tsurf + cs); lss = __ldg(L.lsurf + cs); }
        }
        if (cd != NONE) {
            td = __ldg(L.target + cd);
            ld = __ldg(L.lambda + cd);
            if (surface) { tsd = __ldg(L.tsurf + cd); lsd = __ldg(L.lsurf + cd); }
        }
    }
};

constexpr int PT = 512;            // threads of a pass block; one block per SM
constexpr int PW = PT / 32;        // its warps, an item (a row's segment) each of a chunk
constexpr int UMAX = 4;            // pixels a lane reads at once at most
constexpr int PEND = 3072;         // pending attempts a block lists in shared memory (rounds)
constexpr int PLAN_SMEM = 1024;    // pass plans of up to 1023 histories sit in shared memory
constexpr int CHAIN = 64;          // attempts a cell's list holds
constexpr int TURNS = 64;          // attempts a lane runs before its warp shares out what it holds
constexpr int MAX_ROUNDS = 256;
constexpr uint32_t ROUND_SPAN = MAX_ROUNDS + 2;  // claim tags one pass may use
// passes before the claim tags would overflow 32 bits: the pass that reaches
// it clears the claims and starts the count again
constexpr uint32_t SEQ_LIMIT = 0xFFFFFFFFu / ROUND_SPAN - 1u;
constexpr unsigned long long BARRIER_NS = 2000000000ull;

// Scratch of the passes.  Attempts: a segment of `seg` per block; beside them
// a mailbox and two index words each.  A cell's list: its attempts' count and
// CHAIN entries (priority << 32 | attempt << 2 | only cell << 1 | side), side 0
// for the source.  Claims (rounds): two words per cell (by round parity), each
// (tag << 32 | priority) with the tag (pass sequence x ROUND_SPAN + round)
// rising from pass to pass, so that old claims lose to new ones and nothing
// needs clearing.
struct PassScratch {
    unsigned long long *claim[2];  // ncells each
    void *list;                    // Attempt, or LeanAttempt without chains
    ulonglong2 *mail;              // per attempt
    uint32_t *idx, *link;          // per attempt: the blocks' lists (ready; pending, even rounds) and the lanes'
                                   // stacks (pending, odd rounds)
    uint32_t *count;               // per cell: the attempts listed (zero between passes)
    unsigned long long *chain;     // per cell: CHAIN entries
    uint32_t seg;
    int64_t ncells;
    uint32_t *ctl;                 // CTL_* below, then the pass keys (history x colour)
    const int32_t *vplan;          // each history's first chunk of PW items; vplan[nh]: all chunks; vplan[nh + 1]: the
                                   // pixels a lane of an item reads (useg, 1 to UMAX)
    unsigned long long barrier_ns; // a grid barrier's wait limit
    int32_t withhold;              // a block that never arrives at a barrier (failure tests; -1: none)
    int32_t max_rounds;            // rounds before a pass gives up (CW_ERR_SIMULATION)
};
// control words: the barrier's three 64-bit words (arrivals in the low 16 bits,
// flags summed in the next 16, the blocks' pending attempts summed in the high
// half; used in turn) and the passes' two counts of ready attempts, all cleared
// before every sweep and as the sweep goes on; the error, round and sequence
// records in a line of their own; then the pass keys
enum { CTL_WORDS = 0, CTL_READY = 6, CTL_ERR = 48, CTL_ROUNDS = 49, CTL_SEQ = 50, CTL_KEYS = 64 };

// The n-th barrier of a sweep over the whole (co-resident, cooperatively
// launched) grid; *left: the sum of every block's `pending`, *flags of every
// block's `flag`.  The block's
// writes are ordered before the arrival by the block barrier and the release,
// the others' before what follows by the acquire and the block barrier.  The
// wait gives up after S.barrier_ns; false then, on every thread of the block.
// The block S.withhold (a failure test) never arrives and returns false.
// (Count and arrival in one word: the count apart cost another read of L2 each
// round before any work.)
__device__ __forceinline__ bool grid_barrier(const PassScratch &S, uint32_t n, uint32_t pending, uint32_t flag,
                                             uint32_t *left, uint32_t *flags, uint32_t *s_word) {
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t ok = 1, sum = 0, any = 0;
        if ((int)blockIdx.x == S.withhold) {
            ok = 0;
        } else {
            unsigned long long *w = (unsigned long long *)(S.ctl + CTL_WORDS);
            const unsigned long long mine = 1ull | ((unsigned long long)flag << 16) | ((unsigned long long)pending << 32);
            asm volatile("red.release.gpu.global.add.u64 [%0], %1;" ::"l"(w + n % 3), "l"(mine) : "memory");
            uint32_t spins = 0;
            uint64_t t0 = 0;
            for (;;) {
                unsigned long long v;
                asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(w + n % 3) : "memory");
                if (((uint32_t)v & 0xFFFFu) == gridDim.x) {
                    sum = (uint32_t)(v >> 32);
                    any = ((uint32_t)v >> 16) & 0xFFFFu;
                    break;
                }
                if ((++spins & 255u) == 0) {  // the clock only now and then
                    const uint64_t t = global_ns();
                    if (t0 == 0) t0 = t;
                    else if (t - t0 > S.barrier_ns) { ok = 0; break; }
                }
            }
            // every block has left the barrier before this one
            if (blockIdx.x == 0) w[(n + 2) % 3] = 0ull;
        }
        s_word[0] = ok;
        s_word[1] = sum;
        s_word[2] = any;
    }
    __syncthreads();
    *left = s_word[1];
    *flags = s_word[2];
    return s_word[0] != 0;
}

// This lane's slot (where `take`) in a list counted by *s_n, one shared-memory
// atomic per warp.
__device__ __forceinline__ uint32_t warp_slot(uint32_t *s_n, bool take) {
    const int lane = threadIdx.x & 31;
    const unsigned m = __ballot_sync(0xffffffffu, take);
    uint32_t base = 0;
    if (lane == 0 && m) base = atomicAdd(s_n, (uint32_t)__popc(m));
    base = __shfl_sync(0xffffffffu, base, 0);
    return base + __popc(m & ((1u << lane) - 1u));
}

// The history whose chunks hold chunk vb (plan: nh + 1 prefix of chunks).
__device__ __forceinline__ int plan_find(const int32_t *plan, int nh, int vb) {
    int lo = 0, hi = nh - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (plan[mid] <= vb) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// occupied_span (cpm.rs:774-793) of every volume history, at the start of a
// Monte Carlo step: min and max of x, y, z over the pixels that are not
// medium (the obstacle counts), reduced by blocks (span_blocks); then one
// pixel wider on every side, clipped, or empty (x0 > x1) when all is medium.
__global__ void k_span_reset(int32_t *span, int nh) {
    const int h = blockIdx.x * blockDim.x + threadIdx.x;
    if (h >= nh) return;
    for (int a = 0; a < 3; ++a) {
        span[6 * h + a] = 0x7fffffff;
        span[6 * h + 3 + a] = -1;
    }
}
// (volumes: a plane visits its whole box)
__global__ void k_span_occupied(const int32_t *grid, const int4 *dims, const int64_t *off, const int32_t *blk, int nh,
                                int nblocks, int32_t *span) {
    span_blocks<false>(dims, off, blk, nh, nblocks, span, 6,
                       [&](int h, int64_t i) { return dims[h].z > 1 && grid[i] != 0; });
}
__global__ void k_span_finish(int32_t *span, const int4 *dims, int nh) {
    const int h = blockIdx.x * blockDim.x + threadIdx.x;
    if (h >= nh) return;
    int32_t *s = span + 6 * h;
    if (s[3] < 0) {  // all medium: nothing to visit
        s[0] = 1;
        s[3] = 0;
        return;
    }
    const int lim[3] = {dims[h].x, dims[h].y, dims[h].z};
    for (int a = 0; a < 3; ++a) {
        s[a] = s[a] > 0 ? s[a] - 1 : 0;
        s[3 + a] = s[3 + a] + 1 < lim[a] - 1 ? s[3 + a] + 1 : lim[a] - 1;
    }
}

// Whether items of 32 `useg` pixels, `nvb` chunks of them against `least` of 32,
// give every block four chunks and add no more than an eighth to the slots (a
// history's last chunk is rounded up).
__host__ __device__ __forceinline__ bool useg_pays(int64_t nvb, int64_t least, int useg, int blocks) {
    return nvb * useg * 8 <= least * 9 && nvb >= 4 * blocks;
}

// The pass plan of every volume history from its span: the chunks of PW items
// the largest colour of the span holds, as a prefix over the histories
// (vplan[nh] = all of them), for the largest useg up to `most` that pays.  One
// block: each thread sums a run of histories, the runs' totals are scanned, then
// each run is written.  (With the whole box's useg, a tissue of 84^3 in a box of
// 256^3 had 36 chunks for 148 blocks: 676 us a Monte Carlo step, now 607.)
__global__ void __launch_bounds__(1024) k_pass_plan(const int32_t *span, int nh, int period, int most, int blocks,
                                                    int32_t *vplan) {
    __shared__ int32_t s_run[1024], s_all[UMAX + 1];
    const int per = (nh + blockDim.x - 1) / blockDim.x;
    const int h0 = threadIdx.x * per, h1 = min(h0 + per, nh);
    int useg = 1;
    auto chunks = [&](int h) -> int32_t {
        const int32_t *s = span + 6 * h;
        const int64_t n = colour_items(s[3] - s[0] + 1, s[4] - s[1] + 1, s[5] - s[2] + 1, period, useg);
        return (int32_t)((n + PW - 1) / PW);
    };
    auto mine = [&]() {
        int32_t tot = 0;
        for (int h = h0; h < h1; ++h) tot += chunks(h);
        return tot;
    };
    if (threadIdx.x <= UMAX) s_all[threadIdx.x] = 0;
    __syncthreads();
    for (useg = 1; useg <= most; useg *= 2)
        if (const int32_t tot = mine()) atomicAdd(s_all + useg, tot);
    __syncthreads();
    for (useg = most; useg > 1 && !useg_pays(s_all[useg], s_all[1], useg, blocks);) useg /= 2;
    s_run[threadIdx.x] = mine();
    __syncthreads();
    if (threadIdx.x == 0) {
        vplan[nh + 1] = useg;
        int32_t acc = 0;
        for (int t = 0; t < min(nh, (int)blockDim.x); ++t) {  // (the runs behind are empty)
            const int32_t v = s_run[t];
            s_run[t] = acc;
            acc += v;
        }
        vplan[nh] = acc;
    }
    __syncthreads();
    int32_t acc = s_run[threadIdx.x];
    for (int h = h0; h < h1; ++h) {
        vplan[h] = acc;
        acc += chunks(h);
    }
}

// The acceptance of an attempt: Delta-H <= 0, or u < exp(-Delta-H / T) with
// own_exp.  Its limit, -T ln u taken once before the pass runs, decides all but
// the Delta-H within 1e-10 of it (own_exp, the quotient and the limit are each
// within 1e-14 relatively), which take the exponential: it is a third of an
// attempt's time in the chain of attempts that bounds a pass.  A limit that is
// not a number (u = 0, a temperature that is none) decides nothing.
__device__ __forceinline__ double accept_limit(uint32_t u0, uint32_t u1, double T) {
    const double u = u01(u0, u1);
    return u > 0.0 && T > 0.0 ? -T * log(u) : (double)NAN;
}
__device__ __noinline__ bool accept_exactly(double delta, uint32_t u0, uint32_t u1, double T) {
    return u01(u0, u1) < own_exp(-delta / T);
}
__device__ __forceinline__ bool decide(double delta, double limit, uint32_t u0, uint32_t u1, double T) {
    if (delta <= 0.0) return true;
    const double margin = 1e-10 * (T + limit);
    if (delta < limit - margin) return true;
    if (delta > limit + margin) return false;
    return accept_exactly(delta, u0, u1, T);
}

// A cell's records on their way from one of its attempts to the next: bit 63
// set, the sending attempt's depth (10 bits), the surface (25, signed) and the
// volume (28, signed).  Cells past these ranges take the rounds.
__device__ __forceinline__ unsigned long long pack_records(int32_t vol, int32_t surf, uint32_t depth) {
    return (1ull << 63) | ((unsigned long long)min(depth, 1023u) << 53) | ((unsigned long long)((uint32_t)surf & 0x1FFFFFFu) << 28) |
           (unsigned long long)((uint32_t)vol & 0xFFFFFFFu);
}
__device__ __forceinline__ bool records_fit(int32_t vol, int32_t surf) {
    // (a pass changes a volume by CHAIN at most, a surface by 6 CHAIN)
    return vol > -(1 << 27) + 1024 && vol < (1 << 27) - 1024 && surf > -(1 << 24) + 1024 && surf < (1 << 24) - 1024;
}

struct PassShared {
    double J[64];
    int8_t reach[3 * 124];
    uint32_t word[3], n, pending[2], ready, odd;
    int32_t plan[PLAN_SMEM];
    uint4 edge[PW][64];        // proposals: pixels beside another id, gathered by each warp (x, y: where; z: id);
                               // links: its ready attempts
    uint32_t pend[2][PEND];    // rounds: the pending attempts
};

// One sweep of every colour: a sublattice pass each, one copy attempt at every
// pixel of the pass's colour (the reference's try_flip, cpm.rs:797-838) inside
// each history's box (a volume's occupied span, a plane's whole box), the
// attempts ordered by a per-pass priority and run as that sequence would run
// them.  The pixels of a colour lie outside one another's reach, so two
// attempts meet only through the records of a cell they both involve (volume,
// surface).
//
// Propose: each warp takes items of the colour's pixels (a row's segment, or
// short rows one behind another), a lane up to UMAX pixels at once, and gathers
// those that border another id; 32 of them at a time draw their attempt.  An attempt that copies (source and copied ids
// differ, neither the obstacle) is packed into its block's segment and listed
// with its cells (not the medium).
//
// Link: every attempt finds in its cells' lists the one that follows it (the
// next lower priority) and whether any goes before; the terms the pass cannot
// change are taken.
//
// Run: an attempt that no other goes before on any of its cells runs, and hands
// each cell's records to the attempt that follows there, in that one's mailbox;
// of the two that meet in a mailbox the second finds the first's records and
// runs the attempt.  The last attempt on a cell writes its records.  So every
// attempt runs after all of higher priority that share a cell with it, which
// is the sequence in decreasing priority, whatever the thread schedule, and
// nothing waits: the blocks meet three times a pass, and once more for every
// TURNS attempts that a lane runs in turn.
//
// Rounds: a pass with a cell of more than CHAIN attempts (or records past
// pack_records' ranges), and every pass where there is no room for the lists
// (LEAN), runs by claims: every
// attempt claims its cells with its priority, one that holds all its claims
// runs against the live records, the others claim again, a meeting of the
// blocks between rounds.  The same sequence.
//
// What bounds a pass is its longest chain of attempts that share cells (11 to 36
// of them where cells have 50 to 125 pixels).  A round of claims costs 2 us of
// meeting and two or three reads of L2 in turn, 4-6 us in all; an attempt of a
// chain costs one exchange in L2 with its terms read behind it, about 1 us.
// Large lattices are bound by the attempts' lines, 128 bytes each, in the
// proposals and the terms.  Measured against a launch a pass of rounds only, a
// Monte Carlo step: a 96^3 ball of 125-voxel cells with surfaces (8 passes, 36
// attempts deep) 1,740 -> 574 us, the 256^3 spheroid 1,860 -> 607, a 300 x 300
// tissue (4 sub-sweeps of 2 passes) 990 -> 378, 256 x 256 290 -> 111, the 2048 x
// 2048 cord 820 -> 403, the campaign's 22.3 M pixels 1,520 -> 1,150; dense 4096^2
// and 256^3 lattices as said below.
template <bool LEAN>
__global__ void __launch_bounds__(PT, 1) k_cpm_sweep(LatView L, Tables tabs, int nh, const int32_t *perm,
                                                     const uint32_t *mcs_cur, PassScratch S) {
    // a sweep queued after one that gave up does nothing: the barrier's words,
    // the lists and the claims that one left behind are cleared by the host first
    if (__ldcg(S.ctl + CTL_ERR) != 0u) return;
    __shared__ PassShared P;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int i = threadIdx.x; i < L.K * L.K; i += PT) P.J[i] = tabs.J[i];
    for (int i = threadIdx.x; i < 3 * L.nreach; i += PT) P.reach[i] = tabs.reach[i];
    const bool plan_shared = nh + 2 <= PLAN_SMEM;
    if (plan_shared)
        for (int i = threadIdx.x; i < nh + 2; i += PT) P.plan[i] = S.vplan[i];
    __syncthreads();
    const int32_t *plan = plan_shared ? P.plan : S.vplan;
    const int nvb = plan[nh], useg = plan[nh + 1];
    const uint32_t mcs = *mcs_cur;
    const uint32_t *pass_key = S.ctl + CTL_KEYS;
    const uint32_t id0 = blockIdx.x * S.seg;  // this block's first attempt
    using Record = std::conditional_t<LEAN, LeanAttempt, Attempt>;
    Record *const mine = (Record *)S.list + id0;
    Attempt *const list = (Attempt *)S.list;  // (chains)
    const int h0 = blockIdx.x < nvb ? plan_find(plan, nh, blockIdx.x) : 0;
    uint32_t seq = S.ctl[CTL_SEQ], bar = 0, left = 0, most = 0;
    const bool surf_on = L.surface_on != 0;
    auto gave_up = [&]() {
        if (threadIdx.x == 0) atomicExch(S.ctl + CTL_ERR, 1u);
    };
    for (int pass = 0; pass < L.ncol; ++pass) {
        if (threadIdx.x == 0) P.n = P.ready = P.odd = 0u;
        __syncthreads();
        // ---- propose
        // 32 gathered pixels (those of the lanes with `live`): their attempts
        auto draw = [&](uint4 px, bool live) {
            if (!live) px = make_uint4(0u, 0u, 0u, 0u);
            const int h = (int)(px.x & 0xFFFFu);
            const int x = (int)(px.y & 0xFFFFu), y = (int)(px.y >> 16), z = (int)(px.x >> 16);
            const int4 dm = __ldg(L.dims + h);
            const int64_t off = __ldg(L.off + h);
            const int64_t i = ((int64_t)z * dm.y + y) * dm.x + x;
            const int32_t *g = L.grid + off;
            const uint2 key = __ldg(L.keys + h);
            const uint32_t pkey = __ldcg(pass_key + h * L.ncol + pass);
            // (a batch holds fewer than 2^32 records: their claims alone take 16 bytes each)
            const uint32_t c0 = (uint32_t)__ldg(L.cell_off + h);
            bool copies = live;
            const int32_t src = (int32_t)px.z;
            int32_t dst = 0;
            uint4 r = make_uint4(0, 0, 0, 0);
            // with sub-sweeps, a pixel attempts in this one with probability
            // 1 / subsweeps (its own draw), so that over the Monte Carlo step
            // its attempts are Binomial(subsweeps, 1 / subsweeps), near the
            // Poisson(1) of random pixels
            if (copies && L.take_below && philox((uint32_t)i, mcs, 4u, 0u, key.x, key.y).x >= L.take_below)
                copies = false;
            if (copies) {
                r = philox((uint32_t)i, mcs, 0u, 0u, key.x, key.y);
                int64_t step;
                if (!L.copy_moore) {
                    const Vn vn = vn_of(dm, x, y, z);
                    step = vn.nth((int)(((uint64_t)r.x * (uint64_t)vn.count()) >> 32));
                } else {
                    const Moore mo = moore_of(dm, x, y, z);
                    step = mo.nth((int)(((uint64_t)r.x * (uint64_t)mo.count()) >> 32));
                }
                dst = g[i + step];
                copies = src != dst && dst != OBST;
            }
            const uint32_t e = warp_slot(&P.n, copies);
            if (!copies) return;
            const uint32_t prio = fmix32((uint32_t)i ^ pkey);
            const uint32_t cs = src > 0 ? c0 + (uint32_t)src : NONE, cd = dst > 0 ? c0 + (uint32_t)dst : NONE;
            if constexpr (!LEAN) {
                // both places taken at once
                uint32_t ks = 0, kd = 0;
                if (cs != NONE) ks = atomicAdd(S.count + cs, 1u);
                if (cd != NONE) kd = atomicAdd(S.count + cd, 1u);
                const bool only = cs == NONE || cd == NONE;
                const unsigned long long entry = ((unsigned long long)prio << 32) | ((id0 + e) << 2) | (only ? 2u : 0u);
                if (cs != NONE && ks < CHAIN) S.chain[(size_t)cs * CHAIN + ks] = entry;
                if (cd != NONE && kd < CHAIN) S.chain[(size_t)cd * CHAIN + kd] = entry | 1u;
                if (max(ks, kd) >= CHAIN) P.odd = 1u;
                S.mail[id0 + e] = make_ulonglong2(0ull, 0ull);
            }
            const int64_t gi = off + i;
            if constexpr (LEAN) {
                int4 *const w = (int4 *)(mine + e);
                w[0] = make_int4((int)cs, (int)cd, (int)prio, dst);
                w[1] = make_int4((int)(uint32_t)gi, (int)(gi >> 32), (int)r.y, (int)r.z);
                w[2] = make_int4((int)px.x, (int)px.y, 0, src);
                return;
            }
            int4 *const w = (int4 *)(mine + e);
            w[2] = make_int4(0, 0, (int)cs, (int)cd);
            w[3] = make_int4((int)NONE, (int)NONE, dst, 0);
            w[4] = make_int4((int)(uint32_t)gi, (int)(gi >> 32), (int)r.y, (int)r.z);
            w[6] = make_int4(0, 0, (int)prio, src);
            w[7] = make_int4((int)px.x, (int)px.y, 0, 0);
        };
        {
            uint4 *const gathered = P.edge[warp];
            int have = 0;  // pixels gathered, the same in every lane
            int h = h0;    // a block's chunks come in increasing order: its history only moves forward
            for (int vb = blockIdx.x; vb < nvb; vb += gridDim.x) {
                // (32 histories a step: one at a time, a batch of thousands waited for
                // its plan longer than for its pixels)
                for (int passed = 32; passed == 32; h += passed)
                    passed = __popc(__ballot_sync(0xffffffffu, plan[min(h + 1 + lane, nh)] <= vb));
                const int4 dm = __ldg(L.dims + h);
                int box[6] = {0, 0, 0, dm.x - 1, dm.y - 1, dm.z - 1};
                if (L.span && dm.z > 1)
#pragma unroll
                    for (int a = 0; a < 6; ++a) box[a] = __ldg(L.span + 6 * h + a);
                const uint32_t item = (uint32_t)(vb - plan[h]) * PW + (uint32_t)warp;
                const ColourItems items((uint32_t)(box[3] - box[0] + 1), L.period, useg);
                const ColourRows rows(box, L.period, __ldg(perm + h * L.ncol + pass));
                if (rows.rows == 0u) continue;
                const int32_t *const hist = L.grid + __ldg(L.off + h);
                const int64_t w = dm.x, slice = (int64_t)dm.x * dm.y;
                // every pixel's neighbours read at once (no read waits on another's
                // test); a pixel whose copy neighbours all hold its own id cannot copy
                bool edge[UMAX];
                uint32_t xy[UMAX], hz[UMAX];
                int32_t src[UMAX];
                auto read = [&](auto packed) {
                    constexpr bool PACKED = decltype(packed)::value;
                    const uint32_t k0 = item * 32u * (uint32_t)useg + (uint32_t)lane;
                    uint32_t row = 0, j0 = 0;
                    int x = 0, y = 0, z = 0, fx = 0, nx = 0;
                    if (!PACKED) {
                        row = item / items.segs;
                        j0 = k0 - row * items.segs * 32u * (uint32_t)useg;
                        if (row < rows.rows) rows.at(row, y, z, fx, nx);
                    }
                    // the lane's pixel u into (x, y, z); false without one
                    auto pixel = [&](int u) -> bool {
                        uint32_t j = j0 + 32u * (uint32_t)u;
                        if (PACKED) {
                            row = (k0 + 32u * (uint32_t)u) / items.n;
                            j = k0 + 32u * (uint32_t)u - row * items.n;
                            nx = 0;
                            if (row < rows.rows) rows.at(row, y, z, fx, nx);
                        }
                        x = fx + rows.step * (int)j;
                        return u < useg && (int)j < nx;
                    };
                    if (!L.copy_moore) {
                        int32_t nb[UMAX][6];
                        unsigned there[UMAX];
#pragma unroll
                        for (int u = 0; u < UMAX; ++u) {
                            const bool live = pixel(u);
                            const int32_t *const g = hist + ((int64_t)z * dm.y + y) * dm.x;
                            xy[u] = (uint32_t)x | ((uint32_t)y << 16);
                            hz[u] = (uint32_t)h | ((uint32_t)z << 16);
                            src[u] = OBST;
                            if (live) src[u] = g[x];
                            // (not `: src[u]`: taking the pixel's own id where there is no
                            // neighbour holds every later read until that id has come)
                            const bool has[6] = {live && y > 0, live && y + 1 < dm.y, live && x > 0,
                                                 live && x + 1 < dm.x, live && z > 0, live && z + 1 < dm.z};
                            const int64_t to[6] = {-w, w, -1, 1, -slice, slice};
                            there[u] = 0u;
#pragma unroll
                            for (int q = 0; q < 6; ++q) {
                                nb[u][q] = 0;
                                if (has[q]) {
                                    nb[u][q] = g[x + to[q]];
                                    there[u] |= 1u << q;
                                }
                            }
                        }
#pragma unroll
                        for (int u = 0; u < UMAX; ++u) {
                            edge[u] = false;
#pragma unroll
                            for (int q = 0; q < 6; ++q) edge[u] |= ((there[u] >> q) & 1u) && nb[u][q] != src[u];
                            edge[u] = edge[u] && src[u] != OBST;
                        }
                    } else {
#pragma unroll 1
                        for (int u = 0; u < UMAX; ++u) {
                            bool e = false;
                            int32_t own = OBST;
                            if (pixel(u)) {
                                const int32_t *const g = hist + ((int64_t)z * dm.y + y) * dm.x;
                                own = g[x];
                                const Moore mo = moore_of(dm, x, y, z);
                                if (own != OBST)
                                    for (int q = 0; q < 27; ++q)
                                        if ((mo.mask >> q) & 1u) e |= g[x + mo.step(q)] != own;
                            }
#pragma unroll
                            for (int v = 0; v < UMAX; ++v)
                                if (v == u) {
                                    edge[v] = e;
                                    xy[v] = (uint32_t)x | ((uint32_t)y << 16);
                                    hz[v] = (uint32_t)h | ((uint32_t)z << 16);
                                    src[v] = own;
                                }
                        }
                    }
                };
                if (items.packed) read(std::true_type());
                else read(std::false_type());
#pragma unroll
                for (int u = 0; u < UMAX; ++u) {
                    const unsigned m = __ballot_sync(0xffffffffu, edge[u]);
                    if (edge[u])
                        gathered[have + __popc(m & ((1u << lane) - 1u))] =
                            make_uint4(hz[u], xy[u], (uint32_t)src[u], 0u);
                    have += __popc(m);
                    if (have >= 32) {
                        __syncwarp();
                        const uint4 px = gathered[lane], rest = gathered[32 + lane];
                        __syncwarp();
                        gathered[lane] = rest;
                        have -= 32;
                        draw(px, true);
                        __syncwarp();
                    }
                }
            }
            __syncwarp();
            if (have > 0) draw(gathered[lane], lane < have);
        }
        __syncthreads();
        const uint32_t n = P.n;
        uint32_t flags = 0;
        if (!grid_barrier(S, bar++, n, P.odd, &left, &flags, P.word)) { gave_up(); return; }
        // (the next pass's count: last used by the pass before, which is over)
        if (blockIdx.x == 0 && threadIdx.x == 0) S.ctl[CTL_READY + ((pass + 1) & 1)] = 0u;
        if (left == 0) continue;
        bool linked = !LEAN && flags == 0u;
        const uint32_t tag0 = seq * ROUND_SPAN;  // round r claims with tag tag0 + r
        // round 1's claims
        auto claim_first = [&](const Record &a) {
            const unsigned long long claim = ((unsigned long long)(tag0 + 1u) << 32) | a.prio;
            if (a.cs != NONE) atomicMax(S.claim[1] + a.cs, claim);
            if (a.cd != NONE) atomicMax(S.claim[1] + a.cd, claim);
            if (!LEAN) {
                if (a.cs != NONE) S.count[a.cs] = 0u;
                if (a.cd != NONE) S.count[a.cd] = 0u;
            }
        };
        // ---- link: G lanes of a warp take a cell's whole list, as many cells at once
        // as that leaves room for (a cell waits for its list and then for an
        // exchange; one cell a warp, dense planes of 16.8 M pixels took 2.00 ms a
        // step, now 1.69, and 2.70 -> 1.87 with the nine passes of order 3); each
        // entry's follower into its attempt, and the cell's records to the first
        if constexpr (!LEAN) if (linked) {
            uint32_t *const found = (uint32_t *)P.edge[warp];
            uint32_t have = 0;  // ready attempts found and not yet in the list, the same in every lane
            auto flush = [&](uint32_t m) {
                __syncwarp();
                uint32_t at = 0;
                if (lane == 0) {
                    at = atomicAdd(S.ctl + CTL_READY + (pass & 1), m);
                    atomicAdd(&P.ready, m);
                }
                at = __shfl_sync(0xffffffffu, at, 0);
                if (lane < m) S.idx[at + lane] = found[lane];
                __syncwarp();
            };
            const int64_t stride = (int64_t)gridDim.x * PW;
            // the cells c0 + q stride, `cnt` attempts each (lane q's), for the bits q of `live`
            auto link = [&](auto lanes, unsigned live, uint32_t cnt, int64_t c0) {
                constexpr int G = decltype(lanes)::value;
                const int group = lane / G, gl = lane % G;
                while (live) {
                    int q = -1;  // this group's cell
#pragma unroll
                    for (int g = 0; g < 32 / G; ++g) {
                        if (g == group && live) q = __ffs(live) - 1;
                        live &= live - 1u;
                    }
                    const uint32_t listed = __shfl_sync(0xffffffffu, cnt, q & 31), k = q >= 0 ? listed : 0u;
                    const uint32_t longest = G == 32 ? k : __reduce_max_sync(0xffffffffu, k);
                    const size_t c = q >= 0 ? (size_t)(c0 + q * stride) : 0;
                    const unsigned long long *entries = S.chain + c * CHAIN;
                    const int32_t vol = __ldcg(L.volume + c), surf = surf_on ? __ldcg(L.surface + c) : 0;
                    unsigned long long mine2[2] = {gl < k ? __ldcg(entries + gl) : 0ull, 0ull};
                    if (G == 32 && lane + 32 < k) mine2[1] = __ldcg(entries + 32 + lane);
                    if (k && !records_fit(vol, surf)) P.odd = 1u;
#pragma unroll
                    for (int half = 0; half < (G == 32 ? 2 : 1); ++half) {
                        if (half && k <= 32) break;
                        const unsigned long long own = mine2[half];
                        const uint32_t prio = (uint32_t)(own >> 32);
                        unsigned long long below = 0ull;
                        bool followed = false, first = gl + 32u * half < k;
                        for (uint32_t j = 0; j < longest; ++j) {
                            // (a cell's attempts have distinct priorities)
                            const unsigned long long x =
                                __shfl_sync(0xffffffffu, G < 32 || j < 32 ? mine2[0] : mine2[1], j & 31, G);
                            const uint32_t xp = (uint32_t)(x >> 32);
                            if (G < 32 && j >= k) continue;
                            if (xp > prio) first = false;
                            if (xp < prio && (!followed || x > below)) {
                                below = x;
                                followed = true;
                            }
                        }
                        bool ready = false;
                        const uint32_t id = ((uint32_t)own >> 2);
                        if (gl + 32u * half < k) {
                            if (followed) (own & 1ull ? list[id].next_d : list[id].next_s) = (uint32_t)below;
                            if (first) {
                                const unsigned long long box = pack_records(vol, surf, 0u);
                                unsigned long long met = 0ull;
                                ready = (own & 2ull) != 0ull || (met = atomicExch(&S.mail[id].x, box)) != 0ull;
                                if (ready) S.mail[id] = (own & 1ull) ? make_ulonglong2(met, box) : make_ulonglong2(box, met);
                            }
                        }
                        // (at most one a list)
                        const unsigned some = __ballot_sync(0xffffffffu, ready);
                        if (ready) found[have + __popc(some & ((1u << lane) - 1u))] = id;
                        have += __popc(some);
                        if (have >= 32) {
                            flush(32);
                            const uint32_t rest = found[32 + lane];
                            __syncwarp();
                            found[lane] = rest;
                            have -= 32;
                        }
                    }
                }
            };
            // (a warp's cells lie a stride apart: those with attempts are often the
            // first of the records)
            for (int64_t c0 = blockIdx.x * PW + warp; c0 < S.ncells; c0 += 32 * stride) {
                const uint32_t cnt = c0 + lane * stride < S.ncells ? __ldcg(S.count + c0 + lane * stride) : 0u;
                link(std::integral_constant<int, 4>(), __ballot_sync(0xffffffffu, cnt - 1u < 4u), cnt, c0);
                link(std::integral_constant<int, 8>(), __ballot_sync(0xffffffffu, cnt - 5u < 4u), cnt, c0);
                link(std::integral_constant<int, 16>(), __ballot_sync(0xffffffffu, cnt - 9u < 8u), cnt, c0);
                link(std::integral_constant<int, 32>(), __ballot_sync(0xffffffffu, cnt > 16u), cnt, c0);
            }
            if (have) flush(have);
        }
        // ---- the terms the pass cannot change, over the block's attempts packed
        // together (a contact term reads no pixel of the colour).  Everything is
        // read before anything is written: a write between two reads that it might
        // change holds the second until the first has come.
        for (uint32_t e = threadIdx.x; e < n; e += PT) {
            Record *const a = mine + e;
            if (!linked) claim_first(*a);
            uint32_t cs = 0, cd = 0;
            int32_t dst, src;
            uint2 where, u = make_uint2(0u, 0u);
            if constexpr (LEAN) {
                dst = a->dst;
                src = a->src;
                where = a->where;
            } else {
                const int4 w2 = ((const int4 *)a)[2], w3 = ((const int4 *)a)[3], w4 = ((const int4 *)a)[4],
                           w6 = ((const int4 *)a)[6], w7 = ((const int4 *)a)[7];
                cs = (uint32_t)w2.z;
                cd = (uint32_t)w2.w;
                dst = w3.z;
                src = w6.w;
                where = make_uint2((uint32_t)w7.x, (uint32_t)w7.y);
                u = make_uint2((uint32_t)w4.z, (uint32_t)w4.w);
            }
            const int hh = (int)(where.x & 0xFFFFu);
            const int x = (int)(where.y & 0xFFFFu), y = (int)(where.y >> 16), z = (int)(where.x >> 16);
            const int4 dm = __ldg(L.dims + hh);
            const int64_t c0 = __ldg(L.cell_off + hh), cap = __ldg(L.cell_off + hh + 1) - c0;
            const int64_t i = ((int64_t)z * dm.y + y) * dm.x + x;
            const int32_t *g = L.grid + __ldg(L.off + hh);
            const Vn vn = vn_of(dm, x, y, z);
            int32_t ts = 0, td = 0, tss = 0, tsd = 0;
            double ls = 0.0, ld = 0.0, lss = 0.0, lsd = 0.0;
            if (!LEAN && cs != NONE) {
                ts = __ldg(L.target + cs);
                ls = __ldg(L.lambda + cs);
                if (surf_on) { tss = __ldg(L.tsurf + cs); lss = __ldg(L.lsurf + cs); }
            }
            if (!LEAN && cd != NONE) {
                td = __ldg(L.target + cd);
                ld = __ldg(L.lambda + cd);
                if (surf_on) { tsd = __ldg(L.tsurf + cd); lsd = __ldg(L.lsurf + cd); }
            }
            int32_t ds = 0, dd = 0;
            if (surf_on) surface_change(g, i, vn, src, dst, ds, dd);
            double num;
            const double contact = contact_delta(g, dm, x, y, z, src, dst, L.type + c0, cap, P.J, L.K, P.reach, L.nreach,
                                                 L.across, i, vn, &num);
            const int32_t surfs = (int32_t)((uint32_t)(uint16_t)(int16_t)ds | ((uint32_t)(uint16_t)(int16_t)dd << 16));
            a->dsurf = surfs;
            if constexpr (LEAN) {
                a->contact = contact;
                continue;
            } else {
            const double limit = accept_limit(u.x, u.y, L.temperature);
            ((double2 *)a)[0] = make_double2(contact, limit);
            ((double2 *)a)[1] = make_double2(ls, ld);
            *(int2 *)&a->ts = make_int2(ts, td);
            if (surf_on) {
                ((double2 *)a)[5] = make_double2(lss, lsd);
                *(int2 *)&a->tss = make_int2(tss, tsd);
            }
            }
        }
        __syncthreads();
        if (!grid_barrier(S, bar++, linked ? P.ready : n, P.odd, &left, &flags, P.word)) { gave_up(); return; }
        if (linked && flags != 0u) {
            // a cell's records past the mailboxes' ranges: by rounds
            linked = false;
            for (uint32_t e = threadIdx.x; e < n; e += PT) claim_first(mine[e]);
            if (!grid_barrier(S, bar++, n, 0u, &left, &flags, P.word)) { gave_up(); return; }
        }
        // an attempt on the records given: accepted or not, and its writes
        auto attempt = [&](const Terms &a, int32_t &vs, int32_t &ss, int32_t &vd, int32_t &sd) {
            const bool has_s = a.cs != NONE, has_d = a.cd != NONE;
            const int32_t ds = (int32_t)(int16_t)(a.dsurf & 0xFFFF), dd = (int32_t)(int16_t)(a.dsurf >> 16);
            double delta = a.contact + volume_terms(has_s, vs, a.ts, a.ls, has_d, vd, a.td, a.ld);
            if (surf_on) delta += surface_terms(has_s, ss, a.tss, a.lss, ds, has_d, sd, a.tsd, a.lsd, dd);
            if (!decide(delta, a.limit, a.u0, a.u1, L.temperature)) return false;
            L.grid[a.gi] = a.dst;
            vs -= 1;
            vd += 1;
            ss += ds;
            sd += dd;
            return true;
        };
        if constexpr (!LEAN) if (linked) {
            // ---- run the chains: a lane takes what it made ready, else its spare or
            // its stack, else its next of the list, else another lane's spare
            // (dealt one to a warp, then a second to each: the chains of a warp
            // wait for one another's reads, and its idle lanes take their branches).
            // A warp that has made TURNS puts what it holds back into the list, and
            // the blocks meet and share that out anew: what follows an attempt stays
            // with the warp that ran it, so that of many attempts a few warps came to
            // hold the most (a 256^3 volume of 125-voxel cells, order 1: 2,800 turns
            // for one warp, 42 on average; 10.6 -> 2.7 ms a step).
            const uint32_t warps = gridDim.x * PW, stride = 32u * warps;
            uint32_t begin = 0;  // the list's part that has not been run: [begin, begin + left)
            do {
                if (threadIdx.x == 0) P.ready = 0u;
                __syncthreads();
                const uint32_t end = begin + left;
                uint32_t at = begin + blockIdx.x * PW + warp + lane * warps;
                uint32_t id = NONE, spare = NONE, top = NONE, listed = at < end ? __ldcg(S.idx + at) : NONE;
                // the records that the current attempt and the spare were handed
                unsigned long long box_s = 0ull, box_d = 0ull, spare_s = 0ull, spare_d = 0ull;
                auto stack = [&](uint32_t what, unsigned long long s, unsigned long long d) {
                    S.mail[what] = make_ulonglong2(s, d);
                    S.link[what] = top;
                    top = what;
                };
                for (int turn = 0;; ++turn) {
                    const bool sharing = turn >= TURNS;
                    if (sharing) {
                        // the rest of the warp's part of the list first, so that an
                        // attempt is listed once: as it is linked or as it is put back
                        if (listed != NONE && id != NONE) {
                            stack(id, box_s, box_d);
                            id = NONE;
                        }
                        if (!__any_sync(0xffffffffu, listed != NONE)) {
                            auto put_back = [&](uint32_t what) {
                                const unsigned m = __ballot_sync(0xffffffffu, what != NONE);
                                uint32_t to = 0;
                                if (lane == 0 && m) {
                                    to = atomicAdd(S.ctl + CTL_READY + (pass & 1), (uint32_t)__popc(m));
                                    atomicAdd(&P.ready, (uint32_t)__popc(m));
                                }
                                to = __shfl_sync(0xffffffffu, to, 0) + __popc(m & ((1u << lane) - 1u));
                                if (what != NONE) S.idx[to] = what;
                                return m != 0u;
                            };
                            if (id != NONE) stack(id, box_s, box_d);
                            if (spare != NONE) stack(spare, spare_s, spare_d);
                            while (put_back(top))
                                if (top != NONE) top = S.link[top];
                            break;
                        }
                    }
                    if (id == NONE) {
                        if (spare != NONE && !(sharing && listed != NONE)) {
                            id = spare;
                            box_s = spare_s;
                            box_d = spare_d;
                            spare = NONE;
                        } else if (top != NONE || listed != NONE) {
                            if (top != NONE && !(sharing && listed != NONE)) {
                                id = top;
                                top = S.link[id];
                            } else {
                                id = listed;
                                at += stride;
                                listed = at < end ? __ldcg(S.idx + at) : NONE;
                            }
                            const ulonglong2 b = __ldcg(S.mail + id);
                            box_s = b.x;
                            box_d = b.y;
                        }
                    }
                    const unsigned idle = __ballot_sync(0xffffffffu, id == NONE);
                    if (idle) {
                        const unsigned rich = __ballot_sync(0xffffffffu, spare != NONE), below = (1u << lane) - 1u;
                        if (rich) {
                            const int m = min(__popc(idle), __popc(rich)), ri = __popc(idle & below), rr = __popc(rich & below);
                            const bool takes = ((idle >> lane) & 1u) && ri < m, gives = ((rich >> lane) & 1u) && rr < m;
                            const int from = takes ? (int)__fns(rich, 0, ri + 1) : lane;
                            const uint32_t got = __shfl_sync(0xffffffffu, spare, from);
                            const unsigned long long gs = __shfl_sync(0xffffffffu, spare_s, from),
                                                     gd = __shfl_sync(0xffffffffu, spare_d, from);
                            if (gives) spare = NONE;
                            if (takes) {
                                id = got;
                                box_s = gs;
                                box_d = gd;
                            }
                        } else if (idle == 0xffffffffu) {
                            break;
                        }
                    }
                    if (id != NONE) {
                        Terms a;
                        a.read(list + id, surf_on);
                        const uint32_t cs = a.cs, cd = a.cd;
                        uint32_t depth = 0;
                        int32_t vs = 0, ss = 0, vd = 0, sd = 0;
                        auto open = [&](unsigned long long b, uint32_t c, int32_t &vol, int32_t &surf) {
                            if (c == NONE) return;
                            vol = (int32_t)((uint32_t)b << 4) >> 4;
                            surf = (int32_t)((uint32_t)(b >> 28) << 7) >> 7;
                            depth = max(depth, (uint32_t)(b >> 53) & 1023u);
                        };
                        open(box_s, cs, vs, ss);
                        open(box_d, cd, vd, sd);
                        attempt(a, vs, ss, vd, sd);
                        depth += 1;
                        most = max(most, depth);
                        const uint32_t next[2] = {cs == NONE ? NONE : a.next_s, cd == NONE ? NONE : a.next_d};
                        const unsigned long long send[2] = {pack_records(vs, ss, depth), pack_records(vd, sd, depth)};
                        unsigned long long met[2] = {0ull, 0ull};
#pragma unroll
                        for (int side = 0; side < 2; ++side)
                            if (next[side] != NONE) {
                                const uint32_t to = next[side] >> 2;
                                // its terms into L1 while the exchange is on its way
                                const char *line = (const char *)(list + to);
#pragma unroll
                                for (int q = 0; q < 4; ++q) {
                                    uint32_t t;
                                    if (q < 3 || surf_on) asm volatile("ld.global.u32 %0, [%1];" : "=r"(t) : "l"(line + 32 * q) : "memory");
                                }
                                if (!(next[side] & 2u)) met[side] = atomicExch(&S.mail[to].x, send[side]);
                            }
                        // the last attempt on a cell writes its records
                        if (cs != NONE && next[0] == NONE) {
                            L.volume[cs] = vs;
                            if (surf_on) L.surface[cs] = ss;
                            S.count[cs] = 0u;
                        }
                        if (cd != NONE && next[1] == NONE) {
                            L.volume[cd] = vd;
                            if (surf_on) L.surface[cd] = sd;
                            S.count[cd] = 0u;
                        }
                        id = NONE;
#pragma unroll
                        for (int side = 0; side < 2; ++side) {
                            if (next[side] == NONE || !((next[side] & 2u) || met[side])) continue;
                            const uint32_t to = next[side] >> 2;
                            const unsigned long long bs = (next[side] & 1u) ? met[side] : send[side],
                                                     bd = (next[side] & 1u) ? send[side] : met[side];
                            if (id == NONE) {
                                id = to;
                                box_s = bs;
                                box_d = bd;
                            } else {
                                if (spare != NONE) stack(spare, spare_s, spare_d);
                                spare = to;
                                spare_s = bs;
                                spare_d = bd;
                            }
                        }
                    }
                    __syncwarp();
                }
                begin = end;
                __syncthreads();
                if (!grid_barrier(S, bar++, P.ready, 0u, &left, &flags, P.word)) { gave_up(); return; }
            } while (left != 0u);
            continue;
        }
        // ---- rounds
        const bool listed = n <= PEND;
        uint32_t *const gpend[2] = {S.idx + id0, S.link + id0};
        uint32_t npend = n;  // this block's attempts entering the round
        for (uint32_t r = 1; left != 0; ++r) {
            if ((int)r > S.max_rounds) {
                if (blockIdx.x == 0 && threadIdx.x == 0) atomicExch(S.ctl + CTL_ERR, 2u);
                return;
            }
            most = max(most, r);
            if (threadIdx.x == 0) P.pending[r & 1] = 0u;
            __syncthreads();
            const unsigned long long *cl = S.claim[r & 1];
            unsigned long long *next = S.claim[(r + 1) & 1];
            const uint32_t *pin = listed ? P.pend[(r - 1) & 1] : gpend[(r - 1) & 1];
            uint32_t *pout = listed ? P.pend[r & 1] : gpend[r & 1];
            for (uint32_t e0 = 0; e0 < npend; e0 += PT) {
                const uint32_t e = e0 + threadIdx.x;
                const bool has = e < npend;
                const uint32_t k = has ? (r == 1 ? e : pin[e]) : 0u;
                bool again = false;
                if (has) {
                    const Record &a = mine[k];
                    const unsigned long long key = ((unsigned long long)(tag0 + r) << 32) | a.prio;
                    unsigned long long ks = key, kd = key;
                    if (a.cs != NONE) ks = __ldcg(cl + a.cs);
                    if (a.cd != NONE) kd = __ldcg(cl + a.cd);
                    if (ks == key && kd == key) {
                        int32_t vs = 0, ss = 0, vd = 0, sd = 0;
                        if (a.cs != NONE) { vs = L.volume[a.cs]; if (surf_on) ss = L.surface[a.cs]; }
                        if (a.cd != NONE) { vd = L.volume[a.cd]; if (surf_on) sd = L.surface[a.cd]; }
                        Terms t;
                        if constexpr (LEAN) t.read(&a, L, surf_on);
                        else t.read(&a, surf_on);
                        if (attempt(t, vs, ss, vd, sd)) {
                            // the records: its cells are its own this round
                            if (a.cs != NONE) { L.volume[a.cs] = vs; if (surf_on) L.surface[a.cs] = ss; }
                            if (a.cd != NONE) { L.volume[a.cd] = vd; if (surf_on) L.surface[a.cd] = sd; }
                        }
                    } else {
                        const unsigned long long claim = ((unsigned long long)(tag0 + r + 1u) << 32) | a.prio;
                        if (a.cs != NONE) atomicMax(next + a.cs, claim);
                        if (a.cd != NONE) atomicMax(next + a.cd, claim);
                        again = true;
                    }
                }
                const uint32_t slot = warp_slot(&P.pending[r & 1], again);
                if (again) pout[slot] = k;
            }
            __syncthreads();
            npend = P.pending[r & 1];
            if (!grid_barrier(S, bar++, npend, 0u, &left, &flags, P.word)) { gave_up(); return; }
        }
        // the pass is over on every block: the sequence advances; at its limit
        // the claims are cleared and it starts again
        seq += 1u;
        if (seq >= SEQ_LIMIT) {
            for (int64_t c = (int64_t)blockIdx.x * PT + threadIdx.x; c < S.ncells; c += (int64_t)gridDim.x * PT)
                S.claim[0][c] = S.claim[1][c] = 0ull;
            seq = 0u;
            if (!grid_barrier(S, bar++, 0u, 0u, &left, &flags, P.word)) { gave_up(); return; }
        }
    }
    // the others read the sequence as they started: all have met since
    if (blockIdx.x == 0 && threadIdx.x == 0) S.ctl[CTL_SEQ] = seq;
    most = __reduce_max_sync(0xffffffffu, most);
    if (lane == 0 && most) {
        atomicMax(S.ctl + CTL_ROUNDS, most);
        // (past the limit the sequence has still run whole)
        if ((int)most > S.max_rounds) atomicExch(S.ctl + CTL_ERR, 2u);
    }
}


// The first staged pixel of histories h0..h1 (n sites from `a`) whose id is
// below -1 or at least its history's cell capacity, as an offset from `a`.
__global__ void k_check_ids(const int32_t *stage, int64_t a, int64_t n, const int64_t *off, const int64_t *cell_off,
                            int h0, int h1, unsigned long long *first_bad) {
    const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const int64_t i = a + k;
    int lo = h0, hi = h1;
    while (lo < hi) { const int mid = (lo + hi + 1) >> 1; if (off[mid] <= i) lo = mid; else hi = mid - 1; }
    const int32_t v = stage[i];
    if (v < -1 || (int64_t)v >= cell_off[lo + 1] - cell_off[lo]) atomicMin(first_bad, (unsigned long long)k);
}

__global__ void k_delta_h(LatView L, Tables tabs, int h, int64_t n, const int64_t *site, const int32_t *dstv,
                          double *out) {
    __shared__ double sJ[64];
    __shared__ int8_t sreach[3 * 124];
    for (int i = threadIdx.x; i < L.K * L.K; i += blockDim.x) sJ[i] = tabs.J[i];
    for (int i = threadIdx.x; i < 3 * L.nreach; i += blockDim.x) sreach[i] = tabs.reach[i];
    __syncthreads();
    int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= n) return;
    const int4 dm = L.dims[h];
    const int64_t c0 = L.cell_off[h], cap = L.cell_off[h + 1] - c0;
    const int32_t *g = L.grid + L.off[h];
    int64_t i = site[q];
    int x = (int)(i % dm.x), y = (int)((i / dm.x) % dm.y), z = (int)(i / ((int64_t)dm.x * dm.y));
    const Vn vn = vn_of(dm, x, y, z);
    int32_t src = g[i], dst = dstv[q];
    double num;
    double c = contact_delta(g, dm, x, y, z, src, dst, L.type + c0, cap, sJ, L.K, sreach, L.nreach, L.across, i, vn,
                             &num);
    double v = volume_delta(L.volume, L.target, L.lambda, c0, src, dst);
    double s = 0.0;
    if (L.surface_on) {
        int32_t ds, dd;
        surface_change(g, i, vn, src, dst, ds, dd);
        s = surface_delta(L.surface, L.tsurf, L.lsurf, c0, src, dst, ds, dd);
    }
    double *o = out + 6 * q;
    o[0] = num; o[1] = c; o[2] = v; o[3] = s; o[4] = c + v; o[5] = (c + v) + s;
}

// Recount volumes (and surfaces) from the grid: recount, cpm.rs:1262-1270.
__global__ void k_recount(const int32_t *grid, const int4 *dims, const int64_t *off, const int64_t *cell_off,
                          const int32_t *blk, int nh, int32_t *vol, int32_t *surf) {
    __shared__ int s_h;
    if (threadIdx.x == 0) s_h = plan_history(blk, nh, blockIdx.x);
    __syncthreads();
    int h = s_h;
    int64_t local = (int64_t)(blockIdx.x - blk[h]) * blockDim.x + threadIdx.x;
    if (local >= off[h + 1] - off[h]) return;
    const int32_t *g = grid + off[h];
    int32_t id = g[local];
    int64_t cap = cell_off[h + 1] - cell_off[h];
    if (id < 0 || id >= cap) return;
    atomicAdd(vol + cell_off[h] + id, 1);
    if (surf && id > 0) {
        const int4 dm = dims[h];
        int x = (int)(local % dm.x), y = (int)((local / dm.x) % dm.y), z = (int)(local / ((int64_t)dm.x * dm.y));
        const Vn vn = vn_of(dm, x, y, z);
        int c = 0;
#pragma unroll
        for (int k = 0; k < 6; ++k)
            if (vn.has(k)) c += g[local + vn.step(k)] != id;
        if (c) atomicAdd(surf + cell_off[h] + id, c);
    }
}

__global__ void k_compare(const int32_t *a, const int32_t *b, const int64_t *cell_off, int h, int *bad) {
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    int64_t c0 = cell_off[h], n = cell_off[h + 1] - c0;
    if (i >= 1 && i < n && a[c0 + i] != b[c0 + i]) atomicAdd(bad, 1);
}

// set_contact_order, cpm.rs:274-301.
int make_reach(int order, bool volume, int8_t *off, double *across) {
    *across = 1.0;
    if (order <= 1) return 0;
    int deep = volume ? 2 : 0;
    std::vector<std::array<int, 3>> cand;
    std::vector<int64_t> dist;
    for (int dz = -deep; dz <= deep; ++dz)
        for (int dy = -2; dy <= 2; ++dy)
            for (int dx = -2; dx <= 2; ++dx) {
                if (dx == 0 && dy == 0 && dz == 0) continue;
                cand.push_back({dx, dy, dz});
                dist.push_back((int64_t)dx * dx + dy * dy + dz * dz);
            }
    std::vector<int64_t> u = dist;
    std::sort(u.begin(), u.end());
    u.erase(std::unique(u.begin(), u.end()), u.end());
    int64_t limit = u[std::min<size_t>((size_t)(order - 1), u.size() - 1)];
    int n = 0;
    int64_t acr = 0;
    for (size_t i = 0; i < cand.size(); ++i)
        if (dist[i] <= limit) {
            for (int a = 0; a < 3; ++a) off[3 * n + a] = (int8_t)cand[i][a];
            acr += std::max(cand[i][0], 0);
            ++n;
        }
    *across = (double)acr;
    return n;
}

}  // namespace

int cw_lattice_s::build_plans() {
    ++plans;
    bool volume = g.d[0] > 1;
    nreach = make_reach(order, volume, reach, &across);
    if (nreach == 0 && !copy_moore) {
        period = 0;
        ncol = 2;
    } else if (nreach == 0) {
        // face contact with diagonal copies: a copy's source must not be a
        // pixel of the same colour, so the chessboard gives way to period 2
        period = 2;
        ncol = volume ? 8 : 4;
    } else {
        int r = 1;
        for (int k = 0; k < 3 * nreach; ++k) r = std::max(r, (int)std::abs(reach[k]));
        period = r + 1;
        ncol = volume ? period * period * period : period * period;
    }
    int rc;
    if (pass_grid == 0) {
        int per_sm = 0, dev = 0, nsm = 0;
        CW_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, (const void *)k_cpm_sweep<false>, PT, 0));
        CW_CUDA(cudaGetDevice(&dev));
        CW_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
        pass_grid = std::max(1, per_sm > 0 ? nsm : 0);
    }
    // the pass plan: chunks of PW items, as many as the largest colour of each
    // history's box holds (a plane's plan; in a volume a bound of the plan the
    // device takes from the occupied span every Monte Carlo step).  A lane of an
    // item reads the most pixels (4, 2 or 1) that pay.
    std::vector<int32_t> vp(g.nh + 2, 0);
    auto chunks = [&](int per) -> int64_t {
        for (uint32_t k = 0; k < g.nh; ++k) {
            const int64_t items = colour_items(g.w[k], g.h[k], g.d[k], period, per);
            vp[k + 1] = vp[k] + (int32_t)((items + PW - 1) / PW);
        }
        return vp[g.nh];
    };
    const int64_t least = chunks(1);
    for (useg = UMAX; useg > 1 && !useg_pays(chunks(useg), least, useg, pass_grid);) useg /= 2;
    // the pass scratch: a block's segment holds every pixel of the chunks it
    // visits, (chunks / blocks launched, rounded up) items of 32 useg, in a volume
    // for every useg that a span may be given
    pass_blocks = (int)std::max<int64_t>(1, std::min<int64_t>(volume ? least : chunks(useg), pass_grid));
    pass_seg = 0;
    for (int u = volume ? 1 : useg; u <= useg; u *= 2)
        pass_seg = std::max(pass_seg, (chunks(u) + pass_blocks - 1) / pass_blocks * PW * 32 * u);
    vp[g.nh + 1] = useg;  // (the chunks are useg's: the last counted)
    if (!d_vplan && (rc = dalloc(&d_vplan, (size_t)g.nh + 2)) != CW_OK) return rc;
    CW_CUDA(cudaMemcpyAsync(d_vplan, vp.data(), sizeof(int32_t) * (g.nh + 2), cudaMemcpyHostToDevice, stream()));
    if (!pctl) {
        if ((rc = dalloc(&pctl, CTL_KEYS + 27 * (size_t)g.nh)) != CW_OK) return rc;
        CW_CUDA(cudaMemsetAsync(pctl, 0, sizeof(uint32_t) * (CTL_KEYS + 27 * (size_t)g.nh), stream()));
    }
    CW_CUDA(cudaStreamSynchronize(stream()));
    return CW_OK;
}

// The passes' scratch, taken by the first sweep (a lattice is made with the
// chessboard's plan, twice the pixels of a colour that the contact set on it
// usually has).
int cw_lattice_s::ensure_scratch() {
    int rc;
    if (!claim) {
        if ((rc = dalloc(&claim, 2 * (size_t)ncells)) != CW_OK) return rc;
        CW_CUDA(cudaMemsetAsync(claim, 0, sizeof(unsigned long long) * 2 * (size_t)ncells, stream()));
    }
    const int64_t need = (int64_t)pass_blocks * pass_seg;
    if (need <= plist_cap) return CW_OK;
    ++plans;
    dfree(plist);
    dfree(pidx);
    dfree(pmail);
    plist_cap = 0;
    // By chains: 152 bytes a pixel slot of a colour, and the cells' lists, 516
    // bytes a record, where all this is at most a quarter of the memory that is
    // free (and a list's entry can number the attempts).  Else, or where it could
    // not be had, by rounds: 56 bytes a slot, as fast within a twentieth on large
    // lattices (3.79 ms a step of 33.6 M pixels against 3.61) and half as fast on
    // small ones.
    const size_t chains = (sizeof(Attempt) + sizeof(ulonglong2) + 2 * sizeof(uint32_t)) * (size_t)need;
    const size_t lists = pchain ? 0 : (CHAIN * sizeof(unsigned long long) + sizeof(uint32_t)) * (size_t)ncells;
    size_t unused = 0, whole = 0;
    CW_CUDA(cudaMemGetInfo(&unused, &whole));
    lean = need >= (1ll << 30) || chains + lists > unused / 4;
    if (!lean) {
        auto take = [](auto **p, size_t n) {
            return *p || cudaMalloc((void **)p, sizeof(**p) * n) == cudaSuccess;
        };
        const bool counts = pcount == nullptr;
        if (take(&plist, sizeof(Attempt) / sizeof(uint4) * (size_t)need) && take(&pidx, 2 * (size_t)need) &&
            take(&pmail, (size_t)need) && take(&pcount, (size_t)ncells) && take(&pchain, CHAIN * (size_t)ncells)) {
            if (counts) CW_CUDA(cudaMemsetAsync(pcount, 0, sizeof(uint32_t) * (size_t)ncells, stream()));
            plist_cap = need;
            return CW_OK;
        }
        (void)cudaGetLastError();
        lean = true;
        dfree(plist);
        dfree(pidx);
        dfree(pmail);
    }
    dfree(pcount);
    dfree(pchain);
    if ((rc = dalloc(&plist, sizeof(LeanAttempt) / sizeof(uint4) * (size_t)need)) != CW_OK) return rc;
    if ((rc = dalloc(&pidx, 2 * (size_t)need)) != CW_OK) return rc;
    plist_cap = need;
    return CW_OK;
}

namespace {
struct LatExtra {
    uint32_t *mcs_ctr = nullptr, *mcs_cur = nullptr;
    int32_t *perm = nullptr;
};
}  // namespace

static LatView lat_view(cw_lattice_s *l) {
    LatView v;
    v.grid = l->grid; v.type = l->type; v.volume = l->volume; v.vsnap = l->vsnap; v.target = l->target;
    v.lambda = l->lambda; v.surface = l->surface; v.ssnap = l->ssnap; v.tsurf = l->tsurf; v.lsurf = l->lsurf;
    v.dims = l->g.d_dims; v.off = l->g.d_off; v.cell_off = l->d_cell_off; v.keys = l->d_keys;
    v.K = l->K; v.nreach = l->nreach; v.period = l->period; v.ncol = l->ncol; v.across = l->across;
    v.temperature = l->temperature; v.surface_on = l->surface_on ? 1 : 0; v.copy_moore = l->copy_moore ? 1 : 0;
    v.take_below = l->subsweeps > 1 ? (uint32_t)(4294967296.0 / (double)l->subsweeps) : 0u;
    v.span = l->d_span;
    return v;
}

static Tables lat_tables(const cw_lattice_s *l) {
    Tables t;
    std::memcpy(t.J, l->J, sizeof t.J);
    std::memcpy(t.reach, l->reach, sizeof t.reach);
    return t;
}

// mcs counter (2 words) and colour permutations live in d_flag's neighbours
struct LatDevice {
    uint32_t *mcs;   // [0] counter, [1] current
    int32_t *perm;   // nh * 27
};
static LatDevice dev_of(cw_lattice_s *l) {
    LatDevice d;
    d.mcs = (uint32_t *)l->d_flag;
    d.perm = l->d_flag + 4;
    return d;
}

namespace cw {
int lattice_recount_surfaces(cw_lattice_s *l) {
    Plan &p = l->site_plan;
    if (p.nblocks == 0) {
        std::vector<int64_t> per(l->g.nh);
        for (uint32_t k = 0; k < l->g.nh; ++k) per[k] = l->g.sites(k);
        int rc = p.build(per, T);
        if (rc != CW_OK) return rc;
    }
    CW_CUDA(cudaMemsetAsync(l->vsnap, 0, sizeof(int32_t) * l->ncells, stream()));
    CW_CUDA(cudaMemsetAsync(l->surface, 0, sizeof(int32_t) * l->ncells, stream()));
    k_recount<<<p.nblocks, T, 0, stream()>>>(l->grid, l->g.d_dims, l->g.d_off, l->d_cell_off, p.d_blk, l->g.nh,
                                             l->vsnap, l->surface);
    CW_LAUNCHED();
    return CW_OK;
}

int lattice_recount(cw_lattice_s *l, int32_t *vol_out, int32_t *surf_out) {
    std::vector<int64_t> per(l->g.nh);
    for (uint32_t k = 0; k < l->g.nh; ++k) per[k] = l->g.sites(k);
    Plan p;
    int rc = p.build(per, T);
    if (rc != CW_OK) return rc;
    CW_CUDA(cudaMemsetAsync(vol_out, 0, sizeof(int32_t) * l->ncells, stream()));
    if (surf_out) CW_CUDA(cudaMemsetAsync(surf_out, 0, sizeof(int32_t) * l->ncells, stream()));
    k_recount<<<p.nblocks, T, 0, stream()>>>(l->grid, l->g.d_dims, l->g.d_off, l->d_cell_off, p.d_blk, l->g.nh,
                                             vol_out, surf_out);
    CW_LAUNCHED();
    CW_CUDA(cudaStreamSynchronize(stream()));
    p.release();
    return CW_OK;
}

// One Monte Carlo step of every history (no host synchronisation): the
// colour order, then one cooperative launch of every colour's pass.
int lattice_span_enqueue(cw_lattice_s *l) {
    if (!l->d_span) return CW_OK;
    Plan &p = l->site_plan;
    if (p.nblocks == 0) {
        std::vector<int64_t> per(l->g.nh);
        for (uint32_t k = 0; k < l->g.nh; ++k) per[k] = l->g.sites(k);
        int rc = p.build(per, T);
        if (rc != CW_OK) return rc;
    }
    const int nh = (int)l->g.nh;
    k_span_reset<<<(nh + 127) / 128, 128, 0, stream()>>>(l->d_span, nh);
    CW_LAUNCHED();
    k_span_occupied<<<(p.nblocks + SPAN_BLOCKS - 1) / SPAN_BLOCKS, T, 0, stream()>>>(
        l->grid, l->g.d_dims, l->g.d_off, p.d_blk, nh, p.nblocks, l->d_span);
    CW_LAUNCHED();
    k_span_finish<<<(nh + 127) / 128, 128, 0, stream()>>>(l->d_span, l->g.d_dims, nh);
    CW_LAUNCHED();
    k_pass_plan<<<1, 1024, 0, stream()>>>(l->d_span, nh, l->period, l->useg, l->pass_blocks, l->d_vplan);
    CW_LAUNCHED();
    return CW_OK;
}

int lattice_sweep(cw_lattice_s *l) {
    int rc0 = lattice_span_enqueue(l);
    if (rc0 != CW_OK) return rc0;
    for (int s = 0; s < std::max(l->subsweeps, 1); ++s) {
        int rc = lattice_subsweep(l);
        if (rc != CW_OK) return rc;
    }
    l->mcs += 1;
    return CW_OK;
}

// One sweep of every colour (a whole Monte Carlo step with one sub-sweep);
// the device's step counter advances by one per sub-sweep.
int lattice_subsweep(cw_lattice_s *l) {
    const int rc = l->ensure_scratch();
    if (rc != CW_OK) return rc;
    LatDevice d = dev_of(l);
    k_colour_order<<<1, 128, 0, stream()>>>(l->d_keys, l->g.nh, l->ncol, d.mcs, d.mcs + 1, d.perm,
                                            l->pctl + CTL_KEYS, l->pctl + CTL_WORDS);
    CW_LAUNCHED();
    LatView v = lat_view(l);
    Tables t = lat_tables(l);
    PassScratch S;
    S.claim[0] = l->claim;
    S.claim[1] = l->claim + l->ncells;
    S.list = l->plist;
    S.mail = l->pmail;
    S.idx = l->pidx;
    S.link = l->pidx + l->plist_cap;
    S.count = l->pcount;
    S.chain = l->pchain;
    S.seg = (uint32_t)l->pass_seg;
    S.ncells = l->ncells;
    S.ctl = l->pctl;
    S.vplan = l->d_vplan;
    const TestFaults &tf = test_faults();
    S.barrier_ns = tf.wait_ns ? tf.wait_ns : BARRIER_NS;
    S.withhold = tf.withhold_block;
    S.max_rounds = tf.max_rounds > 0 ? tf.max_rounds : MAX_ROUNDS;
    int nh = (int)l->g.nh;
    const uint32_t *cur = d.mcs + 1;
    void *args[] = {&v, &t, &nh, &d.perm, (void *)&cur, &S};
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.gridDim = dim3((unsigned)l->pass_blocks);
    cfg.blockDim = dim3(PT);
    cfg.dynamicSmemBytes = 0;
    cfg.stream = stream();
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    CW_CUDA(cudaLaunchKernelExC(&cfg, l->lean ? (const void *)k_cpm_sweep<true> : (const void *)k_cpm_sweep<false>, args));
    count_launch(1);
    return CW_OK;
}

// CW_ERR_TIMEOUT (or CW_ERR_SIMULATION) if a pass gave up since the last
// call: a grid barrier that waited too long, or more rounds (a deeper chain)
// than allowed.
int lattice_pass_error(cw_lattice_s *l) {
    uint32_t e = 0;
    CW_CUDA(cudaMemcpy(&e, l->pctl + CTL_ERR, sizeof e, cudaMemcpyDeviceToHost));
    if (!e) return CW_OK;
    // a pass that gave up left the barrier's words, its claims and its cells'
    // lists behind: all start again from zero
    CW_CUDA(cudaMemset(l->pctl, 0, sizeof(uint32_t) * CTL_KEYS));
    if (l->claim) CW_CUDA(cudaMemset(l->claim, 0, sizeof(unsigned long long) * 2 * (size_t)l->ncells));
    if (l->pcount) CW_CUDA(cudaMemset(l->pcount, 0, sizeof(uint32_t) * (size_t)l->ncells));
    return e == 1 ? fail(CW_ERR_TIMEOUT, "a sublattice pass waited too long at a grid barrier")
                  : fail(CW_ERR_SIMULATION, "a sublattice pass needed more rounds than allowed");
}
}  // namespace cw

extern "C" {

int cw_lattice_create(uint32_t nh, const uint32_t *w, const uint32_t *h, const uint32_t *d,
                      const uint32_t *cell_capacity, double temperature, cw_lattice *out) {
    *out = nullptr;
    if (nh > 65535) return fail(CW_ERR_CONFIG, "a lattice batch holds at most 65535 histories");
    cw_lattice_s *l = new cw_lattice_s();
    if (l->hs.init() != CW_OK) { delete l; return CW_ERR_CUDA; }
    CW_SCOPE(l);
    int rc = l->g.init(nh, w, h, d);
    if (rc != CW_OK) { delete l; return rc; }
    bool volume = l->g.d[0] > 1;
    for (uint32_t k = 1; k < nh; ++k)
        if ((l->g.d[k] > 1) != volume) {
            l->g.release();
            delete l;
            return fail(CW_ERR_CONFIG, "a batch holds flat lattices or volumes, not both");
        }
    l->cell_off.assign(nh + 1, 0);
    for (uint32_t k = 0; k < nh; ++k) {
        uint32_t cap = std::max<uint32_t>(cell_capacity ? cell_capacity[k] : 1, 1);
        l->cell_off[k + 1] = l->cell_off[k] + cap;
    }
    l->ncells = l->cell_off[nh];
    l->temperature = temperature;
    l->seed.assign(nh, 0);
    int64_t n = l->g.total, nc = l->ncells;
    if ((rc = dalloc(&l->grid, n)) || (rc = dalloc(&l->type, nc)) || (rc = dalloc(&l->volume, nc)) ||
        (rc = dalloc(&l->target, nc)) || (rc = dalloc(&l->lambda, nc)) || (rc = dalloc(&l->vsnap, nc)) ||
        (rc = dalloc(&l->d_cell_off, nh + 1)) || (rc = dalloc(&l->d_keys, nh)) ||
        (rc = dalloc(&l->d_flag, 4 + 27 * (size_t)nh)) || (rc = dalloc(&l->d_used, nh)) ||
        (volume && (rc = dalloc(&l->d_span, 6 * (size_t)nh)))) {
        cw_lattice_destroy(l);
        return rc;
    }
    CW_CUDA(cudaMemsetAsync(l->grid, 0, sizeof(int32_t) * n, stream()));
    CW_CUDA(cudaMemsetAsync(l->type, 0, sizeof(int32_t) * nc, stream()));
    CW_CUDA(cudaMemsetAsync(l->volume, 0, sizeof(int32_t) * nc, stream()));
    CW_CUDA(cudaMemsetAsync(l->target, 0, sizeof(int32_t) * nc, stream()));
    CW_CUDA(cudaMemsetAsync(l->lambda, 0, sizeof(double) * nc, stream()));
    CW_CUDA(cudaMemsetAsync(l->d_keys, 0, sizeof(uint2) * nh, stream()));
    CW_CUDA(cudaMemsetAsync(l->d_flag, 0, sizeof(int32_t) * (4 + 27 * (size_t)nh), stream()));
    l->used.assign(nh, 1);  // the medium's record
    CW_CUDA(cudaMemcpyAsync(l->d_used, l->used.data(), sizeof(int32_t) * nh, cudaMemcpyHostToDevice, stream()));
    CW_CUDA(cudaMemcpyAsync(l->d_cell_off, l->cell_off.data(), sizeof(int64_t) * (nh + 1), cudaMemcpyHostToDevice,
                            stream()));
    l->K = 1;
    l->J[0] = 0.0;
    l->order = 1;
    if ((rc = l->build_plans()) != CW_OK) { cw_lattice_destroy(l); return rc; }
    CW_CUDA(cudaStreamSynchronize(stream()));
    *out = l;
    return CW_OK;
}

int cw_lattice_destroy(cw_lattice l) {
    if (!l) return CW_OK;
    CW_SCOPE(l);
    dfree(l->grid); dfree(l->type); dfree(l->volume); dfree(l->target); dfree(l->lambda); dfree(l->vsnap);
    dfree(l->surface); dfree(l->ssnap); dfree(l->tsurf); dfree(l->lsurf); dfree(l->d_cell_off); dfree(l->d_keys);
    dfree(l->d_flag); dfree(l->claim); dfree(l->plist); dfree(l->pidx);
    dfree(l->pmail); dfree(l->pcount); dfree(l->pchain); dfree(l->d_vplan); dfree(l->pctl); dfree(l->d_used);
    dfree(l->bath_label); dfree(l->bath_mark); dfree(l->stage); dfree(l->d_bad); dfree(l->d_span);
    l->div.release();
    l->site_plan.release();
    l->g.release();
    l->hs.release();
    delete l;
    return CW_OK;
}

int cw_lattice_capacity(cw_lattice l, uint32_t hist, uint32_t *cap) {
    CW_SCOPE(l);
    if (hist >= l->g.nh) return fail(CW_ERR_NOT_FOUND, "no history " + std::to_string(hist));
    *cap = (uint32_t)(l->cell_off[hist + 1] - l->cell_off[hist]);
    return CW_OK;
}

int cw_lattice_pass_rounds(cw_lattice l, uint32_t *rounds) {
    CW_SCOPE(l);
    uint32_t zero = 0;
    CW_CUDA(cudaStreamSynchronize(stream()));
    CW_CUDA(cudaMemcpy(rounds, l->pctl + CTL_ROUNDS, sizeof(uint32_t), cudaMemcpyDeviceToHost));
    CW_CUDA(cudaMemcpy(l->pctl + CTL_ROUNDS, &zero, sizeof zero, cudaMemcpyHostToDevice));
    return CW_OK;
}

int cw_lattice_set_stream(cw_lattice l, void *stream) {
    CW_SCOPE(l);
    return l->hs.set((cudaStream_t)stream);
}

void *cw_lattice_get_stream(cw_lattice l) { return (void *)l->hs.stream; }

const char *cw_lattice_last_error(cw_lattice l) { return l->hs.err.c_str(); }

int cw_lattice_count(cw_lattice l, uint32_t *nh) {
    CW_SCOPE(l);
    *nh = l->g.nh;
    return CW_OK;
}

int cw_lattice_set_contact(cw_lattice l, int32_t K, const double *J, int32_t order) {
    CW_SCOPE(l);
    if (K < 1 || K > 8) return fail(CW_ERR_CONFIG, "the contact table holds 1 to 8 types, got " + std::to_string(K));
    for (int a = 0; a < K; ++a)
        for (int b = 0; b < K; ++b)
            if (!std::isfinite(J[a * K + b]) || J[a * K + b] != J[b * K + a])
                return fail(CW_ERR_CONFIG, "the contact table must be finite and symmetric");
    l->K = K;
    std::memset(l->J, 0, sizeof l->J);
    std::memcpy(l->J, J, sizeof(double) * K * K);
    l->order = order < 1 ? 1 : order;
    return l->build_plans();
}

int cw_lattice_set_copy_nbhd(cw_lattice l, int32_t nbhd) {
    CW_SCOPE(l);
    if (nbhd != CW_COPY_VON_NEUMANN && nbhd != CW_COPY_MOORE)
        return fail(CW_ERR_CONFIG, "copy neighbourhood " + std::to_string(nbhd) + " is neither von Neumann nor Moore");
    l->copy_moore = nbhd == CW_COPY_MOORE;
    return l->build_plans();
}

int cw_lattice_set_subsweeps(cw_lattice l, int32_t subsweeps) {
    CW_SCOPE(l);
    if (subsweeps < 1 || subsweeps > 64) return fail(CW_ERR_CONFIG, "1 to 64 sub-sweeps a Monte Carlo step");
    l->subsweeps = subsweeps;
    return CW_OK;
}

int cw_lattice_set_temperature(cw_lattice l, double temperature) {
    CW_SCOPE(l);
    if (!(temperature > 0.0)) return fail(CW_ERR_CONFIG, "the temperature must be positive");
    l->temperature = temperature;
    return CW_OK;
}

// Histories h0..h1's sites, staged at `off[h0]`, copied into the grid when
// every id lies in [-1, capacity): the host data lands in the staging buffer,
// a kernel records the first pixel that does not, and only a clean upload
// becomes the grid.
static int upload_range(cw_lattice l, uint32_t h0, uint32_t h1, const int32_t *grid) {
    int rc;
    if (!l->stage && ((rc = dalloc(&l->stage, (size_t)l->g.total)) || (rc = dalloc(&l->d_bad, 1)))) return rc;
    const int64_t a = l->g.off[h0], n = l->g.off[h1 + 1] - a;
    const unsigned long long none = ~0ull;
    CW_CUDA(cudaMemcpyAsync(l->stage + a, grid, sizeof(int32_t) * n, cudaMemcpyHostToDevice, stream()));
    CW_CUDA(cudaMemcpyAsync(l->d_bad, &none, sizeof none, cudaMemcpyHostToDevice, stream()));
    k_check_ids<<<(unsigned)((n + T - 1) / T), T, 0, stream()>>>(l->stage, a, n, l->g.d_off, l->d_cell_off, (int)h0,
                                                                 (int)h1, l->d_bad);
    CW_LAUNCHED();
    unsigned long long bad = none;
    CW_CUDA(cudaMemcpyAsync(&bad, l->d_bad, sizeof bad, cudaMemcpyDeviceToHost, stream()));
    CW_CUDA(cudaStreamSynchronize(stream()));
    if (bad != none) {
        uint32_t h = h0;
        while (h < h1 && l->g.off[h + 1] <= a + (int64_t)bad) ++h;
        const int64_t i = a + (int64_t)bad - l->g.off[h];
        return fail(CW_ERR_CONFIG, "pixel " + std::to_string(i) + " holds id " + std::to_string(grid[bad]) +
                                       ", past the history's cell capacity " +
                                       std::to_string(l->cell_off[h + 1] - l->cell_off[h]));
    }
    CW_CUDA(cudaMemcpyAsync(l->grid + a, l->stage + a, sizeof(int32_t) * n, cudaMemcpyDeviceToDevice, stream()));
    return CW_OK;
}

int cw_lattice_upload(cw_lattice l, uint32_t hist, const int32_t *grid) {
    CW_SCOPE(l);
    if (hist >= l->g.nh) return fail(CW_ERR_NOT_FOUND, "no history " + std::to_string(hist));
    return upload_range(l, hist, hist, grid);
}

int cw_lattice_upload_all(cw_lattice l, const int32_t *grids) {
    CW_SCOPE(l);
    if (l->g.nh == 0) return CW_OK;
    return upload_range(l, 0, l->g.nh - 1, grids);
}

int cw_lattice_download(cw_lattice l, uint32_t hist, int32_t *grid) {
    CW_SCOPE(l);
    if (hist >= l->g.nh) return fail(CW_ERR_NOT_FOUND, "no history " + std::to_string(hist));
    CW_CUDA(cudaMemcpyAsync(grid, l->grid + l->g.off[hist], sizeof(int32_t) * l->g.sites(hist), cudaMemcpyDeviceToHost,
                            stream()));
    CW_CUDA(cudaStreamSynchronize(stream()));
    return CW_OK;
}

int cw_lattice_download_all(cw_lattice l, int32_t *grids) {
    CW_SCOPE(l);
    CW_CUDA(cudaMemcpyAsync(grids, l->grid, sizeof(int32_t) * l->g.total, cudaMemcpyDeviceToHost, stream()));
    CW_CUDA(cudaStreamSynchronize(stream()));
    return CW_OK;
}

static int check_cells(cw_lattice l, uint32_t hist, uint32_t n) {
    if (hist >= l->g.nh) return fail(CW_ERR_NOT_FOUND, "no history " + std::to_string(hist));
    if ((int64_t)n > l->cell_off[hist + 1] - l->cell_off[hist])
        return fail(CW_ERR_CONFIG, "more records than the history's cell capacity");
    return CW_OK;
}

int cw_cells_set(cw_lattice l, uint32_t hist, uint32_t n, const int32_t *type, const int32_t *volume,
                 const int32_t *target, const double *lambda) {
    CW_SCOPE(l);
    int rc = check_cells(l, hist, n);
    if (rc != CW_OK) return rc;
    for (uint32_t i = 0; i < n; ++i)
        if (type && (type[i] < 0 || type[i] >= l->K))
            return fail(CW_ERR_CONFIG, "cell " + std::to_string(i) + " has type " + std::to_string(type[i]) +
                                           " outside the contact table");
    int64_t c0 = l->cell_off[hist];
    if ((int32_t)n > l->used[hist]) {
        l->used[hist] = (int32_t)n;
        CW_CUDA(cudaMemcpyAsync(l->d_used + hist, &l->used[hist], sizeof(int32_t), cudaMemcpyHostToDevice, stream()));
    }
    if (type) CW_CUDA(cudaMemcpyAsync(l->type + c0, type, 4 * n, cudaMemcpyHostToDevice, stream()));
    if (volume) CW_CUDA(cudaMemcpyAsync(l->volume + c0, volume, 4 * n, cudaMemcpyHostToDevice, stream()));
    if (target) CW_CUDA(cudaMemcpyAsync(l->target + c0, target, 4 * n, cudaMemcpyHostToDevice, stream()));
    if (lambda) CW_CUDA(cudaMemcpyAsync(l->lambda + c0, lambda, 8 * n, cudaMemcpyHostToDevice, stream()));
    CW_CUDA(cudaStreamSynchronize(stream()));
    return CW_OK;
}

int cw_cells_get(cw_lattice l, uint32_t hist, uint32_t n, int32_t *type, int32_t *volume, int32_t *target,
                 double *lambda) {
    CW_SCOPE(l);
    int rc = check_cells(l, hist, n);
    if (rc != CW_OK) return rc;
    int64_t c0 = l->cell_off[hist];
    if (type) CW_CUDA(cudaMemcpyAsync(type, l->type + c0, 4 * n, cudaMemcpyDeviceToHost, stream()));
    if (volume) CW_CUDA(cudaMemcpyAsync(volume, l->volume + c0, 4 * n, cudaMemcpyDeviceToHost, stream()));
    if (target) CW_CUDA(cudaMemcpyAsync(target, l->target + c0, 4 * n, cudaMemcpyDeviceToHost, stream()));
    if (lambda) CW_CUDA(cudaMemcpyAsync(lambda, l->lambda + c0, 8 * n, cudaMemcpyDeviceToHost, stream()));
    CW_CUDA(cudaStreamSynchronize(stream()));
    return CW_OK;
}

int cw_cells_set_surface(cw_lattice l, uint32_t hist, uint32_t n, const int32_t *target_surface,
                         const double *lambda_surface) {
    CW_SCOPE(l);
    int rc = check_cells(l, hist, n);
    if (rc != CW_OK) return rc;
    if (!l->surface_on) {
        int64_t nc = l->ncells;
        if ((rc = dalloc(&l->surface, nc)) || (rc = dalloc(&l->ssnap, nc)) || (rc = dalloc(&l->tsurf, nc)) ||
            (rc = dalloc(&l->lsurf, nc)))
            return rc;
        CW_CUDA(cudaMemsetAsync(l->tsurf, 0, 4 * nc, stream()));
        CW_CUDA(cudaMemsetAsync(l->lsurf, 0, 8 * nc, stream()));
        l->surface_on = true;
    }
    int64_t c0 = l->cell_off[hist];
    CW_CUDA(cudaMemcpyAsync(l->tsurf + c0, target_surface, 4 * n, cudaMemcpyHostToDevice, stream()));
    CW_CUDA(cudaMemcpyAsync(l->lsurf + c0, lambda_surface, 8 * n, cudaMemcpyHostToDevice, stream()));
    return lattice_recount(l, l->vsnap, l->surface);  // vsnap is scratch until the next pass
}

int cw_cells_get_surface(cw_lattice l, uint32_t hist, uint32_t n, int32_t *surface) {
    CW_SCOPE(l);
    int rc = check_cells(l, hist, n);
    if (rc != CW_OK) return rc;
    if (!l->surface_on) return fail(CW_ERR_NOT_FOUND, "the surface constraint is off");
    CW_CUDA(cudaMemcpyAsync(surface, l->surface + l->cell_off[hist], 4 * n, cudaMemcpyDeviceToHost, stream()));
    CW_CUDA(cudaStreamSynchronize(stream()));
    return CW_OK;
}

int cw_lattice_set_seed(cw_lattice l, uint32_t hist, uint64_t seed) {
    CW_SCOPE(l);
    if (hist >= l->g.nh) return fail(CW_ERR_NOT_FOUND, "no history " + std::to_string(hist));
    l->seed[hist] = seed;
    uint2 k = make_uint2((uint32_t)seed, (uint32_t)(seed >> 32));
    CW_CUDA(cudaMemcpyAsync(l->d_keys + hist, &k, sizeof k, cudaMemcpyHostToDevice, stream()));
    CW_CUDA(cudaStreamSynchronize(stream()));
    return CW_OK;
}

int cw_lattice_set_mcs(cw_lattice l, uint32_t mcs) {
    CW_SCOPE(l);
    l->mcs = mcs;
    // the draws count sub-sweeps
    const uint32_t eff = mcs * (uint32_t)std::max(l->subsweeps, 1);
    CW_CUDA(cudaMemcpyAsync(l->d_flag, &eff, sizeof eff, cudaMemcpyHostToDevice, stream()));
    CW_CUDA(cudaStreamSynchronize(stream()));
    return CW_OK;
}

int cw_lattice_get_mcs(cw_lattice l, uint32_t *mcs) {
    CW_SCOPE(l);
    *mcs = l->mcs;
    return CW_OK;
}

int cw_lattice_mcs(cw_lattice l, uint32_t sweeps) {
    CW_SCOPE(l);
    for (uint32_t s = 0; s < sweeps; ++s) {
        int rc = lattice_sweep(l);
        if (rc != CW_OK) return rc;
    }
    CW_CUDA(cudaStreamSynchronize(stream()));
    return lattice_pass_error(l);
}

int cw_lattice_delta_h_batch(cw_lattice l, uint32_t hist, uint32_t n, const int64_t *site, const int32_t *dst,
                             double *out) {
    CW_SCOPE(l);
    if (hist >= l->g.nh) return fail(CW_ERR_NOT_FOUND, "no history " + std::to_string(hist));
    if (n == 0) return CW_OK;
    int64_t ns = l->g.sites(hist), cap = l->cell_off[hist + 1] - l->cell_off[hist];
    for (uint32_t q = 0; q < n; ++q)
        if (site[q] < 0 || site[q] >= ns || dst[q] < -1 || dst[q] >= cap)
            return fail(CW_ERR_CONFIG, "proposal " + std::to_string(q) + " is outside the lattice or the records");
    int64_t *d_site;
    int32_t *d_dst;
    double *d_out;
    int rc;
    if ((rc = dalloc(&d_site, n)) || (rc = dalloc(&d_dst, n)) || (rc = dalloc(&d_out, 6 * (size_t)n))) return rc;
    CW_CUDA(cudaMemcpyAsync(d_site, site, 8 * (size_t)n, cudaMemcpyHostToDevice, stream()));
    CW_CUDA(cudaMemcpyAsync(d_dst, dst, 4 * (size_t)n, cudaMemcpyHostToDevice, stream()));
    k_delta_h<<<(n + T - 1) / T, T, 0, stream()>>>(lat_view(l), lat_tables(l), (int)hist, n, d_site, d_dst, d_out);
    CW_LAUNCHED();
    CW_CUDA(cudaMemcpyAsync(out, d_out, 48 * (size_t)n, cudaMemcpyDeviceToHost, stream()));
    CW_CUDA(cudaStreamSynchronize(stream()));
    dfree(d_site); dfree(d_dst); dfree(d_out);
    return CW_OK;
}

int cw_lattice_verify(cw_lattice l, uint32_t hist, int32_t *ok) {
    CW_SCOPE(l);
    if (hist >= l->g.nh) return fail(CW_ERR_NOT_FOUND, "no history " + std::to_string(hist));
    int32_t *vol, *surf = nullptr;
    int *bad;
    int rc;
    if ((rc = dalloc(&vol, l->ncells)) || (rc = dalloc(&bad, 1))) return rc;
    if (l->surface_on && (rc = dalloc(&surf, l->ncells)) != CW_OK) return rc;
    if ((rc = lattice_recount(l, vol, surf)) != CW_OK) return rc;
    CW_CUDA(cudaMemsetAsync(bad, 0, sizeof(int), stream()));
    int64_t cap = l->cell_off[hist + 1] - l->cell_off[hist];
    unsigned nb = (unsigned)((cap + T - 1) / T);
    k_compare<<<nb, T, 0, stream()>>>(vol, l->volume, l->d_cell_off, (int)hist, bad);
    CW_LAUNCHED();
    if (surf) {
        k_compare<<<nb, T, 0, stream()>>>(surf, l->surface, l->d_cell_off, (int)hist, bad);
        CW_LAUNCHED();
    }
    int hbad = 0;
    CW_CUDA(cudaMemcpyAsync(&hbad, bad, sizeof(int), cudaMemcpyDeviceToHost, stream()));
    CW_CUDA(cudaStreamSynchronize(stream()));
    *ok = hbad == 0;
    dfree(vol); dfree(bad); dfree(surf);
    return CW_OK;
}

}  // extern "C"
