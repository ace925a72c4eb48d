// The FP64 relax of small fields kept on chip: the reference's red-black SOR
// (relax / sor_sweep / half_sweep, pde.rs:245-405) pixel for pixel, its values
// and sweep counts to the bit, in one cooperative launch a solve.
//
// What bounds a small field's relax is not its bytes (a 301 x 287 plane is
// 0.7 MB) but what stands between two half-sweeps: with one launch a
// half-sweep and one a stop test, a sweep took three launches and 10 us on that
// plane, and up to 256 sweeps were queued past the one that settled.  Here the span of a history's free pixels is cut into one tile per
// block, every block resident (one per SM); a block holds its tile with a
// halo in shared memory, its coefficients for the whole solve, and runs K
// half-sweeps on it between two meetings of the history's blocks, at which it
// writes its interior out, reads its halo anew and learns the largest change
// of each sweep.  Within a round every window pixel is updated; the error of
// a window edge inside the history moves in one ring per half-sweep, so after
// K of them the interior, K + 1 away from it, and the ring around the
// interior are what K half-sweeps of the whole history give (the argument of
// field32.cu's windows).  A round in which sweep s settled is taken again from
// its start for s sweeps only, so that the field and the count are the
// reference's although K half-sweeps ran.  Measured (B200): that plane 10.0 ->
// 1.20 us a sweep, a 256 x 256 sheet with a first-order sink stopping on the
// residual 14 -> 1.8 us, a ball's 40^3 free voxels 10 -> 5.3 us.
//
// A pixel's arithmetic is k_sor64_half's, operation for operation.  Its
// quotient t / den is the one place that differs: den never changes during a
// solve, so its reciprocal y = 1 / den is taken once and the quotient is
// corrected with it, q += y (t - q den) twice from q = t y.  With y the rounded
// reciprocal and the residual formed exactly by a fused multiply-add, the
// first step leaves q within an ulp and the second rounds it as the division
// does (Markstein, "Computation of elementary functions on the IBM RISC
// System/6000 processor", IBM J. Res. Dev. 34, 1990, theorem on the final
// quotient step), as long as nothing leaves the range of normal numbers: a t
// or den outside 2^+-600, 2^+-200 (a zero t among them) is divided.
// This file is built without fused multiply-add contraction.
#include <algorithm>
#include <cmath>
#include <cstddef>
#include <type_traits>

#include "cw_internal.cuh"
#include "field_kernels.cuh"

using namespace cw;

namespace {

constexpr int RT = 512;          // the most threads of a block
constexpr int NW = RT / 32;
constexpr int MAX_K = 16;        // half-sweeps between two meetings
constexpr int MAX_S = MAX_K / 2;
constexpr int SLOTS = 2 * MAX_S; // a round's words: the largest change and the largest residual of each sweep
constexpr int SMEM_MAX = 220 * 1024;
constexpr unsigned long long WAIT_NS = 2000000000ull;
constexpr long long LAUNCH_SWEEPS = 16384;  // the most sweeps one launch takes; a solve that needs more is launched again

// One history's tiling: its swept box, the tiles along each axis, the window
// sizes they need, and its first block.
struct Part {
    int32_t h, first, nblocks;
    int32_t lo[3], n[3];   // the span of the free pixels: origin and sides
    int32_t g[3];          // tiles along x, y, z
    int32_t k;             // half-sweeps a round (even)
    int32_t most;          // volumes: pixels of a colour in its largest window
    int64_t shift;         // pixel i of the batch stands at other[i - shift]
};

struct Args {
    FieldView fv;
    double *other;                // the second buffer of the exchange: of each history the run of pixels that its
                                  // windows read
    const Part *parts;
    int nparts;
    RelaxState *st;
    long long max_sweeps;
    uint32_t *arrivals;           // per history: its blocks' meetings, counted up
    unsigned long long *slots;    // per history: three sets of SLOTS words, in turn
    uint32_t *failed;             // set by a block whose meeting did not end in time
    unsigned long long wait_ns;
    int withhold;                 // a block that never arrives at a meeting (failure tests; -1: none)
};

// The largest over a warp of non-negative doubles' bits, on every lane: the high
// words first, then the low words of those that hold the largest.
__device__ __forceinline__ unsigned long long warp_max_bits(unsigned long long b) {
    const unsigned hi = (unsigned)(b >> 32), top = __reduce_max_sync(0xffffffffu, hi);
    const unsigned lo = __reduce_max_sync(0xffffffffu, hi == top ? (unsigned)b : 0u);
    return ((unsigned long long)top << 32) | lo;
}

__device__ __forceinline__ double2 with_reciprocal(double den) {
    const unsigned e = ((unsigned)__double2hiint(den) >> 20) & 0x7ffu;
    const bool fine = den > 0.0 && e - (1023u - 200u) <= 400u;
    return make_double2(den, fine ? 1.0 / den : 0.0);
}

__device__ __forceinline__ unsigned high_word(double v) { return (unsigned)__double2hiint(v); }

// |b - A c| of a pixel as the stop counts it (k_residual64): none where the
// floor holds an empty pixel down.
__device__ __forceinline__ double projected_residual(double t, double den, double cv, bool floor) {
    const double r = t - den * cv;
    return (floor && cv <= 0.0 && r < 0.0) ? 0.0 : fabs(r);
}

// The larger of `most` and a non-negative v, as bits; a NaN counts for nothing,
// as in fmax.
__device__ __forceinline__ unsigned long long larger_bits(unsigned long long most, double v) {
    if (!(v > 0.0)) return most;
    const unsigned long long b = (unsigned long long)__double_as_longlong(v);
    return b > most ? b : most;
}

// U pixels of one colour: k_sor64_half's update of those in `free` on their
// d sum + sources t and (den, 1 / den) dn, the largest change of those in
// `inner` and (RES) their largest residual, of black pixels after the update,
// of red ones before it.  The comparisons of the usual case are made on the
// doubles' bits (an FP64 compare and select takes the pipe 3.5 times as long as
// an addition); what they do not order as FP64 does, a quotient outside the
// corrected range, an infinity or a NaN, is taken again by division and fmax.
template <int U, bool RES>
__device__ __forceinline__ void relax_pixels(const double (&t)[U], const double2 (&dn)[U], const double (&before)[U],
                                             unsigned free, unsigned inner, bool black, double om, double omc,
                                             bool floor, double (&after)[U], unsigned long long &moved,
                                             unsigned long long &worst) {
    constexpr unsigned EXP = 0x7ff00000u;
    unsigned odd = 0;
    unsigned long long change[U], res[U];
#pragma unroll
    for (int j = 0; j < U; ++j) {
        double q = t[j] * dn[j].y;
        q = fma(fma(-q, dn[j].x, t[j]), dn[j].y, q);
        q = fma(fma(-q, dn[j].x, t[j]), dn[j].y, q);
        double v = omc * before[j] + om * q;
        if (floor && (int)high_word(v) < 0) v = 0.0;
        after[j] = v;
        change[j] = (unsigned long long)__double_as_longlong(v - before[j]) & 0x7fffffffffffffffull;
        bool o = (high_word(t[j]) << 1) - ((1023u - 600u) << 21) > (1200u << 21) || high_word(dn[j].y) == 0u ||
                 (unsigned)(change[j] >> 32) >= EXP;
        if (RES) {
            const double cv = black ? v : before[j];
            const double r = t[j] - dn[j].x * cv;
            const bool empty = floor && (long long)__double_as_longlong(cv) <= 0ll && (int)high_word(r) < 0;
            res[j] = empty ? 0ull : (unsigned long long)__double_as_longlong(r) & 0x7fffffffffffffffull;
            o = o || (unsigned)(res[j] >> 32) >= EXP;
        }
        if (o) odd |= 1u << j;
    }
    odd &= free;
    if (odd) {
#pragma unroll
        for (int j = 0; j < U; ++j) {
            if (!((odd >> j) & 1u)) continue;
            const double q = t[j] / dn[j].x;
            double v = omc * before[j] + om * q;
            if (floor) v = fmax(v, 0.0);
            after[j] = v;
            change[j] = larger_bits(0ull, fabs(v - before[j]));
            if (RES) res[j] = larger_bits(0ull, projected_residual(t[j], dn[j].x, black ? v : before[j], floor));
        }
    }
#pragma unroll
    for (int j = 0; j < U; ++j) {
        if (!((free >> j) & 1u)) after[j] = before[j];
        if ((inner >> j) & 1u) {
            moved = change[j] > moved ? change[j] : moved;
            if (RES) worst = res[j] > worst ? res[j] : worst;
        }
    }
}

// The meeting of a history's blocks: the n-th ends when all have arrived n
// times.  Bounded: false when it did not end in time, and on the block `withhold`,
// which does not arrive.
__device__ __forceinline__ bool meet(uint32_t *arrivals, uint32_t target, unsigned long long wait_ns, int withhold,
                                     int *s_ok) {
    __syncthreads();
    if (threadIdx.x == 0 && (int)blockIdx.x == withhold) {
        *s_ok = 0;
    } else if (threadIdx.x == 0) {
        int ok = 1;
        // the block's writes, ordered before this thread by the barrier, are
        // released with the arrival; the acquiring load and the barrier behind
        // it order the other blocks' writes before what follows
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(arrivals) : "memory");
        uint32_t spins = 0;
        uint64_t t0 = 0;
        while ((int32_t)(ld_acquire_gpu(arrivals) - target) < 0) {
            if ((++spins & 255u) == 0) {
                const uint64_t t = global_ns();
                if (t0 == 0) t0 = t;
                else if (t - t0 > wait_ns) { ok = 0; break; }
            }
        }
        *s_ok = ok;
    }
    __syncthreads();
    return *s_ok != 0;
}

// What a block's round leaves: each warp's maxima of each sweep, the
// history's maxima, and whether the meeting ended.
struct Rounds {
    unsigned long long part[SLOTS][NW], all[SLOTS];
    int ok;
};

// The block's history: the last part that begins at or before it.
__device__ __forceinline__ Part part_of(const Args &a) {
    int q = 0;
    while (q + 1 < a.nparts && a.parts[q + 1].first <= (int)blockIdx.x) ++q;
    return a.parts[q];
}

// A history's solve, by all its blocks: rounds of pt.k half-sweeps and a
// meeting.  load(src, halo): the window's pixels (halo: all but the interior's
// free ones) from a buffer, ready to be swept when it returns; store(dst): the
// interior's free ones out to a buffer; sweep(n): n sweeps of the window, each warp's
// maxima into S.part (the changes, then from MAX_S the residuals) before its
// last block barrier or this function's first; worst(): the interior's
// largest residual.
template <bool RES, class Load, class Store, class Sweep, class Worst>
__device__ __forceinline__ void solve_rounds(const Args &a, const Part &pt, Load load, Store store, Sweep sweep,
                                             Worst worst, Rounds &S) {
    const int tid = threadIdx.x, nw = blockDim.x >> 5, h = pt.h, b = (int)blockIdx.x - pt.first;
    const double tol = a.st[h].tol;
    uint32_t *arrivals = a.arrivals + h;
    unsigned long long *slots = a.slots + (size_t)h * 3 * SLOTS;
    double *const other = a.other - pt.shift;
    long long taken = 0;
    uint32_t meetings = 0;
    int cur = 0, settled = 0;
    double change = 0.0, resid = 0.0;
    auto met = [&]() -> bool {
        if (meet(arrivals, (uint32_t)pt.nblocks * ++meetings, a.wait_ns, a.withhold, &S.ok)) return true;
        if (tid == 0) atomicExch(a.failed, 1u);
        return false;
    };
    for (int round = 0; taken < a.max_sweeps; ++round) {
        const int n = (int)min((long long)(pt.k / 2), a.max_sweeps - taken);
        sweep(n);
        store(cur ? a.fv.c : other);
        __syncthreads();
        unsigned long long *set = slots + (round % 3) * SLOTS;
        if (tid < SLOTS && ((tid < n) || (RES && tid >= MAX_S && tid - MAX_S < n))) {
            unsigned long long m = 0ull;
            for (int w = 0; w < nw; ++w) m = max(m, S.part[tid][w]);
            if (m) atomicMax(set + tid, m);
        }
        if (!met()) return;
        if (tid < SLOTS) S.all[tid] = __ldcg(set + tid);
        // last read before the meeting that has just ended
        if (b == 0 && tid < SLOTS) slots[((round + 2) % 3) * SLOTS + tid] = 0ull;
        load(cur ? a.fv.c : other, true);
        int s = 0;
        for (; s < n; ++s) {
            change = __longlong_as_double((long long)S.all[s]);
            if (RES) resid = __longlong_as_double((long long)S.all[MAX_S + s]);
            if ((RES ? resid : change) < tol) {
                settled = 1;
                break;
            }
        }
        const int kept = settled ? s + 1 : n;
        taken += kept;
        if (settled && kept < n) {
            // the round again from its start, as far as the sweep that settled;
            // where that start is the field itself, every block has read it
            // before any writes it
            load(cur ? other : a.fv.c, false);
            if (cur == 0 && !met()) return;
            sweep(kept);
            store(a.fv.c);
            break;
        }
        cur ^= 1;
        if (settled || taken >= a.max_sweeps) {
            if (cur != 0) store(a.fv.c);  // the round's start was read before the meeting
            break;
        }
    }
    if (!RES) {
        // the residual of the field as it is left, for the report
        const unsigned long long m = warp_max_bits(worst());
        if ((tid & 31) == 0 && m) atomicMax(&a.st[h].resid, m);
    }
    if (b == 0 && tid == 0) {
        // the other blocks read `done` as they start: all have met since
        RelaxState &s = a.st[h];
        s.sweeps += taken;
        s.last_change = change;
        if (RES) s.last_resid = resid;
        s.done = settled;
    }
}

// ------------------------------------------------------------------ planes
//
// Windows of 2 G columns held in registers: a lane has a pair of columns (x
// even and odd, one pixel of each colour a row) over R rows, G lanes a strip
// of R rows, 32 / G strips a warp.  A pixel's neighbours are in the lane's own
// registers but one along x (a shuffle) and, in a strip's first and last rows,
// one along y (the neighbouring strip's row, published in shared memory after
// every half-sweep).  Windows start at even x and y.  A window's outermost
// pixels never change (held, or outside the box) or lie K + 1 or more from the
// interior, so what the shuffles and the missing rows bring them does not
// matter; a pixel outside the box is kept at zero, as a missing neighbour
// counts.  GEN: first-order sinks, production, or free pixels on the box's
// border, whose (den, 1 / den) and production are read from shared memory; else
// every free pixel has four neighbours and one denominator.
template <int G, int R, bool RES, bool GEN>
__global__ void __launch_bounds__(RT, 1) k_relax64_plane(Args a) {
    extern __shared__ __align__(16) unsigned char sm[];
    __shared__ Rounds S;
    const Part pt = part_of(a);
    const int h = pt.h;
    if (a.st[h].done) return;  // the history's every block: settled in an earlier launch
    const FieldView &fv = a.fv;
    const int4 dm = fv.dims[h];
    const int64_t off = fv.off[h];
    const int H = pt.k + 1, b = (int)blockIdx.x - pt.first;
    const int at[2] = {b % pt.g[0], b / pt.g[0]};
    int in0[2], in1[2], w0[2];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        in0[k] = pt.lo[k] + (int)((int64_t)pt.n[k] * at[k] / pt.g[k]);
        in1[k] = pt.lo[k] + (int)((int64_t)pt.n[k] * (at[k] + 1) / pt.g[k]);
        // beyond the span every pixel is held: one ring of them is enough
        w0[k] = max(in0[k] - H, pt.lo[k] - 1) & ~1;
    }
    const int tid = threadIdx.x, lane32 = tid & 31, warp = tid >> 5;
    const int lane = tid % G, strip = tid / G, strips = (int)blockDim.x / G;
    const int gx = w0[0] + 2 * lane, gy0 = w0[1] + strip * R;
    // published rows: [first or last of the strip][column of the pair][strip + 1][lane],
    // a row of zeros before the first strip and behind the last
    double *const edge = (double *)sm;
    const int eab = (strips + 2) * G, eside = 2 * eab;
    double2 *const dy = (double2 *)(edge + 2 * eside);      // GEN: [row of the strip][column][thread]
    const int per = 2 * R * (int)blockDim.x;                 // pixels of the window
    double *const pr = (double *)(dy + (GEN ? per : 0));
    // the uptake in registers, but for the tallest strips
    constexpr bool UP_REG = R <= 4;
    double *const up = pr + (GEN && fv.pr ? per : 0);
    for (int p = tid; p < 2 * eside; p += blockDim.x) edge[p] = 0.0;
    double va[R], vb[R], ua[UP_REG ? R : 1], ub[UP_REG ? R : 1];
    unsigned free_a = 0, free_b = 0, inner_a = 0, inner_b = 0;
    const bool inx = gx < dm.x && gx >= 0, inx1 = gx + 1 < dm.x && gx + 1 >= 0;
#pragma unroll
    for (int j = 0; j < R; ++j) {
        const int gy = gy0 + j;
        const bool iny = gy >= 0 && gy < dm.y, rin = gy >= in0[1] && gy < in1[1];
        const int64_t i = off + (int64_t)gy * dm.x + gx;
        if (iny && inx && !fv.held[i]) free_a |= 1u << j;
        if (iny && inx1 && !fv.held[i + 1]) free_b |= 1u << j;
        if (fv.up) {
            const double u0 = (free_a >> j) & 1u ? fv.up[i] : 0.0, u1 = (free_b >> j) & 1u ? fv.up[i + 1] : 0.0;
            if (UP_REG) {
                ua[UP_REG ? j : 0] = u0;
                ub[UP_REG ? j : 0] = u1;
            } else {
                up[2 * j * (int)blockDim.x + tid] = u0;
                up[(2 * j + 1) * (int)blockDim.x + tid] = u1;
            }
        }
        if (rin && gx >= in0[0] && gx < in1[0]) inner_a |= free_a & (1u << j);
        if (rin && gx + 1 >= in0[0] && gx + 1 < in1[0]) inner_b |= free_b & (1u << j);
        if (GEN) {
            const double ry = (gy > 0 ? 1.0 : 0.0) + (gy + 1 < dm.y ? 1.0 : 0.0);
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                double2 dn = make_double2(1.0, 1.0);
                double p = 0.0;
                if (((e ? free_b : free_a) >> j) & 1u) {
                    const double real = ry + (gx + e > 0 ? 1.0 : 0.0) + (gx + e + 1 < dm.x ? 1.0 : 0.0);
                    double den = real * fv.d + fv.decay;
                    if (fv.ks) den = den + fv.ks[i + e];
                    dn = with_reciprocal(den);
                    if (fv.pr) p = fv.pr[i + e];
                }
                dy[(2 * j + e) * (int)blockDim.x + tid] = dn;
                if (fv.pr) pr[(2 * j + e) * (int)blockDim.x + tid] = p;
            }
        }
    }
    const double2 dy4 = with_reciprocal(4.0 * fv.d + fv.decay);
    const double om = a.st[h].omega, omc = 1.0 - om, d = fv.d, source = fv.source;
    const bool floor = fv.floor, has_pr = GEN && fv.pr != nullptr, has_up = fv.up != nullptr;
    double *const my_edge = edge + (strip + 1) * G + lane;
    // the strip's first and last row of one colour (C: first row's column C,
    // last row's column 1 - C)
    auto publish = [&](int c) {
        my_edge[c * eab] = c ? vb[0] : va[0];
        my_edge[eside + (1 - c) * eab] = c ? va[R - 1] : vb[R - 1];
    };
    auto load = [&](const double *src, bool halo) {
#pragma unroll
        for (int j = 0; j < R; ++j) {
            const int gy = gy0 + j;
            const double *p = src + off + (int64_t)gy * dm.x + gx;
            const bool iny = gy >= 0 && gy < dm.y;
            if (!(halo && ((inner_a >> j) & 1u))) va[j] = iny && inx ? __ldcg(p) : 0.0;
            if (!(halo && ((inner_b >> j) & 1u))) vb[j] = iny && inx1 ? __ldcg(p + 1) : 0.0;
        }
        publish(0);
        publish(1);
        __syncthreads();
    };
    auto store = [&](double *dst) {
#pragma unroll
        for (int j = 0; j < R; ++j) {
            double *p = dst + off + (int64_t)(gy0 + j) * dm.x + gx;
            if ((inner_a >> j) & 1u) p[0] = va[j];
            if ((inner_b >> j) & 1u) p[1] = vb[j];
        }
    };
    // row j's pixel of colour C is the pair's column (C + j) mod 2; d sum +
    // sources of each row's pixel of the colour, add_sources' order on
    // pixel_sums64's sum
    auto gather = [&](auto colour, double (&t)[R], double2 (&dn)[R]) {
        constexpr int C = decltype(colour)::value;
        double side[R];
#pragma unroll
        for (int j = 0; j < R; ++j)
            side[j] = ((C + j) & 1) == 0 ? __shfl_up_sync(0xffffffffu, vb[j], 1, G)
                                         : __shfl_down_sync(0xffffffffu, va[j], 1, G);
        // above the first row: the last row of the strip before, same column;
        // below the last row: the first row of the strip behind
        const double above = my_edge[eside + C * eab - G], below = my_edge[(1 - C) * eab + G];
#pragma unroll
        for (int j = 0; j < R; ++j) {
            const bool even = ((C + j) & 1) == 0;
            double sum = even ? side[j] + vb[j] : va[j] + side[j];
            const double ym = j > 0 ? (even ? va[j > 0 ? j - 1 : 0] : vb[j > 0 ? j - 1 : 0]) : above;
            const double yp = j < R - 1 ? (even ? va[j < R - 1 ? j + 1 : j] : vb[j < R - 1 ? j + 1 : j]) : below;
            sum = sum + ym;
            sum = sum + yp;
            const int k = (2 * j + (even ? 0 : 1)) * (int)blockDim.x + tid;
            dn[j] = GEN ? dy[k] : dy4;
            t[j] = d * sum;
            t[j] = t[j] + source;
            if (has_pr) t[j] = t[j] + pr[k];
            if (has_up) t[j] = t[j] - (UP_REG ? (even ? ua[UP_REG ? j : 0] : ub[UP_REG ? j : 0]) : up[k]);
        }
    };
    // one half-sweep
    auto half = [&](auto colour, unsigned long long &moved, unsigned long long &worst) {
        constexpr int C = decltype(colour)::value;
        double t[R], before[R], after[R];
        double2 dn[R];
        gather(colour, t, dn);
#pragma unroll
        for (int j = 0; j < R; ++j) before[j] = ((C + j) & 1) == 0 ? va[j] : vb[j];
        // the rows whose pixel of this colour is the pair's first column
        constexpr unsigned FIRST = C == 0 ? 0x55u : 0xaau;
        relax_pixels<R, RES>(t, dn, before, (free_a & FIRST) | (free_b & ~FIRST), (inner_a & FIRST) | (inner_b & ~FIRST),
                             C == 1, om, omc, floor, after, moved, worst);
#pragma unroll
        for (int j = 0; j < R; ++j) {
            if (((C + j) & 1) == 0) va[j] = after[j];
            else vb[j] = after[j];
        }
        publish(C);
    };
    auto residual = [&](auto colour, unsigned long long &worst) {
        constexpr int C = decltype(colour)::value;
        double t[R];
        double2 dn[R];
        gather(colour, t, dn);
#pragma unroll
        for (int j = 0; j < R; ++j) {
            const bool even = ((C + j) & 1) == 0;
            if (((even ? inner_a : inner_b) >> j) & 1u)
                worst = larger_bits(worst, projected_residual(t[j], dn[j].x, even ? va[j] : vb[j], floor));
        }
    };
    auto record = [&](int slot, unsigned long long x) {
        const unsigned long long m = warp_max_bits(x);
        if (lane32 == 0) S.part[slot][warp] = m;
    };
    using Red = std::integral_constant<int, 0>;
    using Black = std::integral_constant<int, 1>;
    auto sweep = [&](int n) {
        unsigned long long res = 0ull;
        for (int k = 0; k < n; ++k) {
            unsigned long long moved = 0ull, red = 0ull, black = 0ull;
            half(Red(), moved, red);
            __syncthreads();
            half(Black(), moved, black);
            record(k, moved);
            if (RES) {
                // the red residual of the sweep before came with this sweep's red half
                if (k > 0) record(MAX_S + k - 1, res > red ? res : red);
                res = black;
            }
            __syncthreads();
        }
        if (RES) {
            residual(Red(), res);
            record(MAX_S + n - 1, res);
        }
    };
    __syncthreads();  // the published rows' zeros
    load(fv.c, false);
    // the window's held pixels into the other buffer too, before the first meeting
#pragma unroll
    for (int j = 0; j < R; ++j) {
        const int gy = gy0 + j;
        double *p = a.other - pt.shift + off + (int64_t)gy * dm.x + gx;
        const bool iny = gy >= 0 && gy < dm.y;
        if (iny && inx && !((free_a >> j) & 1u)) p[0] = va[j];
        if (iny && inx1 && !((free_b >> j) & 1u)) p[1] = vb[j];
    }
    solve_rounds<RES>(a, pt, load, store, sweep, [&]() {
        unsigned long long worst = 0ull;
        residual(Red(), worst);
        residual(Black(), worst);
        return worst;
    }, S);
}

// ------------------------------------------------------------------ volumes
//
// RES: the stop is the residual's (CW_STOP_RESIDUAL).  P: the most free pixels of a colour a thread has in its window, whose values,
// uptakes and places it keeps in registers for the whole solve; 0: any
// number, read from shared memory each time.
//
// The window's pixels are stored by colour, each row's pixels of a colour side
// by side (entry xh of row y holds x = x0 + 2 xh + s, x0 even, s the parity
// that colour takes in the row), so that a warp's lanes read consecutive words:
// a pixel's neighbours along x are entries xh - 1 + s and xh + s of the other
// colour's row, its neighbours along y and z entry xh of the rows beside it.
// Rows, planes and entries outside the window are kept at zero.  The free
// pixels of each colour are listed once, so that a half-sweep's lanes are all
// at work whatever the tissue's shape.
template <bool RES, int P>
__global__ void __launch_bounds__(RT, 1) k_relax64_volume(Args a) {
    extern __shared__ __align__(16) unsigned char sm[];
    __shared__ double2 s_dy[8];
    __shared__ Rounds S;
    __shared__ int s_count[2];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const Part pt = part_of(a);
    const int h = pt.h;
    if (a.st[h].done) return;  // the history's every block: settled in an earlier launch
    const FieldView &fv = a.fv;
    const int4 dm = fv.dims[h];
    const int64_t off = fv.off[h];
    const int K = pt.k, H = K + 1;
    const int b = (int)blockIdx.x - pt.first;
    const int at[3] = {b % pt.g[0], (b / pt.g[0]) % pt.g[1], b / (pt.g[0] * pt.g[1])};
    const int side[3] = {dm.x, dm.y, dm.z};
    int in0[3], in1[3], w0[3], wn[3];  // the interior [in0, in1) and the window's origin and sides
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        in0[k] = pt.lo[k] + (int)((int64_t)pt.n[k] * at[k] / pt.g[k]);
        in1[k] = pt.lo[k] + (int)((int64_t)pt.n[k] * (at[k] + 1) / pt.g[k]);
        // beyond the span every pixel is held: one ring of them is enough
        w0[k] = max(max(in0[k] - H, pt.lo[k] - 1), 0);
        const int w1 = min(min(in1[k] + H, pt.lo[k] + pt.n[k] + 1), side[k]);
        if (k == 0) w0[k] &= ~1;
        wn[k] = w1 - w0[k];
    }
    const int hw = (wn[0] + 1) >> 1, stride = hw + 2, zs = (wn[1] + 2) * stride;
    const int nent = (wn[2] + 2) * zs;
    const int nrows = wn[1] * wn[2];
    // shared memory: per-pixel (den, 1/den), values, production, uptake (each
    // array: the red pixels' entries, then the black ones'), the free pixels of
    // each colour, the rows
    double2 *const dy = (double2 *)sm;
    double *const v = (double *)(dy + (fv.ks ? 2 * (size_t)nent : 0));
    double *const pr = v + 2 * (size_t)nent;
    double *const up = pr + (fv.pr ? 2 * (size_t)nent : 0);
    uint32_t *const list = (uint32_t *)(up + (fv.up ? 2 * (size_t)nent : 0));
    int32_t *const site = (int32_t *)(list + 2 * (size_t)nent);  // of each listed pixel, in its history
    uint32_t *const rows = (uint32_t *)(site + 2 * (size_t)nent);
    if (tid < 8) s_dy[tid] = with_reciprocal((double)tid * fv.d + fv.decay);
    if (tid < 2) s_count[tid] = 0;
    for (int p = tid; p < 2 * nent; p += RT) v[p] = 0.0;
    // a row's first entry, its parity (y + z; x0 is even) and whether it is an
    // interior row
    for (int r = tid; r < nrows; r += RT) {
        const int z = r / wn[1], y = r - z * wn[1];
        const int base = (z + 1) * zs + (y + 1) * stride + 1;
        const int gy = w0[1] + y, gz = w0[2] + z;
        const bool inner = gy >= in0[1] && gy < in1[1] && gz >= in0[2] && gz < in1[2];
        rows[r] = ((uint32_t)base << 2) | (uint32_t)(((gy + gz) & 1) << 1) | (inner ? 1u : 0u);
    }
    __syncthreads();
    // the coefficients and the free pixels, once.  A listed pixel: its entry (of
    // both colours' 2 nent), its count of real neighbours from bit 24, bit 30
    // its parity s, bit 31 set in the interior
    for (int r = warp; r < nrows; r += NW) {
        const uint32_t rw = rows[r];
        const int z = r / wn[1], y = r - z * wn[1];
        const int par = (int)((rw >> 1) & 1u), gy = w0[1] + y, gz = w0[2] + z;
        const int32_t row = (gz * dm.y + gy) * dm.x + w0[0];  // a history holds fewer than 2^31 pixels
        const int64_t first = off + row;
        for (int c = 0; c < 2; ++c) {
            const int s = (c + par) & 1;
            for (int x0 = 0; x0 < hw; x0 += 32) {
                const int xh = x0 + lane, x = 2 * xh + s, gx = w0[0] + x;
                const bool in = xh < hw && x < wn[0], free = in && !fv.held[first + x];
                const int e = (c ? nent : 0) + (int)(rw >> 2) + xh;
                if (in) v[e] = __ldcg(fv.c + first + x);
                const unsigned m = __ballot_sync(0xffffffffu, free);
                int from = 0;
                if (lane == 0 && m) from = atomicAdd(&s_count[c], __popc(m));
                from = __shfl_sync(0xffffffffu, from, 0);
                if (!free) continue;
                const int real = (gx > 0) + (gx + 1 < dm.x) + (gy > 0) + (gy + 1 < dm.y) + (gz > 0) + (gz + 1 < dm.z);
                const bool inner = (rw & 1u) && gx >= in0[0] && gx < in1[0];
                const int k = (c ? nent : 0) + from + __popc(m & ((1u << lane) - 1u));
                site[k] = row + x;
                list[k] = (uint32_t)e | ((uint32_t)real << 24) | ((uint32_t)s << 30) | (inner ? 0x80000000u : 0u);
                if (fv.ks) dy[e] = with_reciprocal((double)real * fv.d + fv.decay + fv.ks[first + x]);
                if (fv.pr) pr[e] = fv.pr[first + x];
                if (fv.up) up[e] = fv.up[first + x];
            }
        }
    }
    __syncthreads();

    const double om = a.st[h].omega, omc = 1.0 - om;
    const double d = fv.d, source = fv.source;
    const bool floor = fv.floor, has_ks = fv.ks != nullptr, has_pr = fv.pr != nullptr, has_up = fv.up != nullptr;
    constexpr int ALL = 6;
    const double2 dy_all = s_dy[ALL];  // a pixel with every neighbour real, no first-order sink
    constexpr uint32_t ENTRY = 0xFFFFFFu;
    // d sum + sources of a listed pixel of colour c with uptake u: add_sources'
    // order on pixel_sums64's sum
    auto rhs = [&](int c, uint32_t it, double u) -> double {
        const int e = (int)(it & ENTRY);
        const double *o = v + e + (c ? -nent : nent);
        const double *x = o + (int)((it >> 30) & 1u);
        double sum = x[-1];
        sum = sum + x[0];
        sum = sum + o[-stride];
        sum = sum + o[stride];
        sum = sum + o[-zs];
        sum = sum + o[zs];
        double t = d * sum;
        t = t + source;
        if (has_pr) t = t + pr[e];
        if (has_up) t = t - u;
        return t;
    };
    auto den_of = [&](uint32_t it) -> double2 {
        if (has_ks) return dy[it & ENTRY];
        const int real = (int)((it >> 24) & 7u);
        return real == ALL ? dy_all : s_dy[real];
    };
    // U listed pixels of colour c, those of them that `mine` names
    auto update = [&](int c, auto &it, unsigned mine, auto &cur, auto &u, unsigned long long &moved,
                      unsigned long long &worst) {
        constexpr int U = sizeof(it) / sizeof(it[0]);
        double t[U], after[U];
        double2 dn[U];
        unsigned inner = 0;
#pragma unroll
        for (int j = 0; j < U; ++j) {
            dn[j] = den_of(it[j]);
            t[j] = rhs(c, it[j], u[j]);
            inner |= (it[j] >> 31) << j;
        }
        relax_pixels<U, RES>(t, dn, cur, mine, inner & mine, c == 1, om, omc, floor, after, moved, worst);
#pragma unroll
        for (int j = 0; j < U; ++j)
            if ((mine >> j) & 1u) v[it[j] & ENTRY] = cur[j] = after[j];
    };
    // this thread's listed pixels (P > 0): place, value, uptake; a thread with
    // fewer takes its colour's first one and leaves it as it is
    constexpr int PP = P > 0 ? P : 1;
    uint32_t it0[PP], it1[PP];
    int32_t at0[PP], at1[PP];
    double cur0[PP], cur1[PP], up0[PP], up1[PP];
    unsigned mine0 = 0, mine1 = 0;
    const int count[2] = {s_count[0], s_count[1]};
    auto own = [&](int c, auto &it, auto &place, unsigned &mine, auto &cur, auto &u) {
#pragma unroll
        for (int j = 0; j < PP; ++j) {
            const bool ok = tid + j * RT < count[c];
            if (ok) mine |= 1u << j;
            it[j] = count[c] ? list[(c ? nent : 0) + (ok ? tid + j * RT : 0)]
                             : (uint32_t)((c ? nent : 0) + zs + stride + 1);
            place[j] = ok ? site[(c ? nent : 0) + tid + j * RT] : 0;
            cur[j] = v[it[j] & ENTRY];
            u[j] = has_up && count[c] ? up[it[j] & ENTRY] : 0.0;
        }
    };
    if (P > 0) {
        own(0, it0, at0, mine0, cur0, up0);
        own(1, it1, at1, mine1, cur1, up1);
    }
    auto take = [&](const double *src, bool halo, auto &it, auto &place, unsigned mine, auto &cur) {
#pragma unroll
        for (int j = 0; j < PP; ++j)
            if (((mine >> j) & 1u) && !(halo && (it[j] >> 31))) v[it[j] & ENTRY] = cur[j] = __ldcg(src + place[j]);
    };
    auto load = [&](const double *src, bool halo) {
        src += off;
        if (P > 0) {
            take(src, halo, it0, at0, mine0, cur0);
            take(src, halo, it1, at1, mine1, cur1);
        } else {
            for (int c = 0; c < 2; ++c)
#pragma unroll 4
                for (int k = tid; k < count[c]; k += RT) {
                    const uint32_t it = list[(c ? nent : 0) + k];
                    if (!(halo && (it >> 31))) v[it & ENTRY] = __ldcg(src + site[(c ? nent : 0) + k]);
                }
        }
        __syncthreads();
    };
    auto store = [&](double *dst) {
        dst += off;
        if (P > 0) {
#pragma unroll
            for (int j = 0; j < PP; ++j) {
                if (((mine0 >> j) & 1u) && (it0[j] >> 31)) dst[at0[j]] = cur0[j];
                if (((mine1 >> j) & 1u) && (it1[j] >> 31)) dst[at1[j]] = cur1[j];
            }
        } else {
            for (int c = 0; c < 2; ++c)
                for (int k = tid; k < count[c]; k += RT) {
                    const uint32_t it = list[(c ? nent : 0) + k];
                    if (it >> 31) dst[site[(c ? nent : 0) + k]] = v[it & ENTRY];
                }
        }
    };
    auto half = [&](int c, unsigned long long &moved, unsigned long long &worst) {
        if (P > 0) {
            if (c == 0) update(0, it0, mine0, cur0, up0, moved, worst);
            else update(1, it1, mine1, cur1, up1, moved, worst);
            return;
        }
        constexpr int U = 2;
        for (int k = tid; k < count[c]; k += U * RT) {
            uint32_t it[U];
            double cur[U], u[U];
            unsigned mine = 0;
#pragma unroll
            for (int j = 0; j < U; ++j) {
                const bool ok = k + j * RT < count[c];
                if (ok) mine |= 1u << j;
                it[j] = list[(c ? nent : 0) + (ok ? k + j * RT : k)];
                cur[j] = v[it[j] & ENTRY];
                u[j] = has_up ? up[it[j] & ENTRY] : 0.0;
            }
            update(c, it, mine, cur, u, moved, worst);
        }
    };
    // the largest residual of the interior's pixels of colour c as they stand
    auto residual = [&](int c, unsigned long long &worst) {
        for (int k = tid; k < count[c]; k += RT) {
            const uint32_t it = list[(c ? nent : 0) + k];
            if (!(it >> 31)) continue;
            const int e = (int)(it & ENTRY);
            worst = larger_bits(worst, projected_residual(rhs(c, it, has_up ? up[e] : 0.0), den_of(it).x, v[e], floor));
        }
    };
    auto record = [&](int slot, unsigned long long x) {
        const unsigned long long m = warp_max_bits(x);
        if (lane == 0) S.part[slot][warp] = m;
    };
    // n sweeps on the window as it stands, their maxima into S.part
    auto sweep = [&](int n) {
        unsigned long long res = 0ull;
        for (int k = 0; k < n; ++k) {
            unsigned long long moved = 0ull, red = 0ull, black = 0ull;
            half(0, moved, red);
            __syncthreads();
            half(1, moved, black);
            record(k, moved);
            if (RES) {
                // the red residual of the sweep before came with this sweep's red half
                if (k > 0) record(MAX_S + k - 1, res > red ? res : red);
                res = black;
            }
            __syncthreads();
        }
        if (RES) {
            residual(0, res);
            record(MAX_S + n - 1, res);
        }
    };

    solve_rounds<RES>(a, pt, load, store, sweep, [&]() {
        unsigned long long worst = 0ull;
        residual(0, worst);
        residual(1, worst);
        return worst;
    }, S);
}

// What a history's tiles cost: cycles a sweep, of a meeting with the reload
// behind it (measured 2.0 us, most of it the round trips to L2 of the arrival,
// the wait and the halo) and K half-sweeps.  A half-sweep measured 520 cycles
// at 4 updates a scheduler's warps, 750 at 8, 1,440 at 16 and 3,300 at 32 (GEN
// and the residual's stop half as much again).
constexpr double MEET_CYCLES = 4000.0;

// A plane's windows: 2 G columns, R rows a strip, `threads` threads a block.
// (R = 4 at 128 or 256 threads measured 1.34-1.44 us a sweep on the plane above
// where R = 2 at twice the threads took 1.21-1.27.)
struct Shape {
    int G, R, threads;
};
constexpr Shape SHAPES[] = {{16, 2, 128}, {16, 2, 256}, {16, 2, 512}, {32, 2, 512}, {32, 4, 512}, {32, 8, 512}};

// The rounds and tiles of the least cost for one history under a shape.
double plan_plane(Part &p, int blocks, const Shape &sh, bool gen) {
    const int win[2] = {2 * sh.G, sh.R * (sh.threads / sh.G)};
    const double half = 150.0 + (sh.R > 4 ? 105.0 : 80.0) * (gen ? 1.4 : 1.0) * sh.R * (sh.threads / 128);
    double best = 0.0;
    for (int K = 2; K <= MAX_K; K += 2) {
        int g[2];
        for (int k = 0; k < 2; ++k) {
            // one tile needs the ring beyond the span; else K + 1 pixels on
            // either side; the origin is rounded down to even
            const int most = win[k] - 2 * (K + 1) - 1;
            g[k] = p.n[k] + 3 <= win[k] ? 1 : most >= 1 ? (p.n[k] + most - 1) / most : blocks + 1;
        }
        if ((int64_t)g[0] * g[1] > blocks) continue;
        const double cost = ((g[0] * g[1] == 1 ? 1000.0 : MEET_CYCLES) + K * half) / (K / 2);
        if (best == 0.0 || cost < best) {
            best = cost;
            p.g[0] = g[0];
            p.g[1] = g[1];
            p.g[2] = 1;
            p.k = K;
            p.nblocks = g[0] * g[1];
        }
    }
    return best;
}

size_t plane_smem(const Shape &sh, bool gen, bool pr, bool up) {
    const size_t edge = 4 * (size_t)(sh.threads / sh.G + 2) * sh.G * sizeof(double), per = (size_t)2 * sh.R * sh.threads;
    return edge + per * ((gen ? sizeof(double2) + (pr ? sizeof(double) : 0) : 0) + (up && sh.R > 4 ? sizeof(double) : 0));
}

size_t volume_smem(const int (&wn)[3], bool ks, bool pr, bool up) {
    const size_t hw = (wn[0] + 2) / 2, zs = (size_t)(wn[1] + 2) * (hw + 2), nent = (size_t)(wn[2] + 2) * zs;
    return nent * 2 * (8 + 4 + 4 + (ks ? 16 : 0) + (pr ? 8 : 0) + (up ? 8 : 0)) + 4 * (size_t)wn[1] * wn[2];
}

// The same for a volume, with the shared memory it needs; 0: no tiling fits.
double plan_volume(Part &p, int blocks, bool ks, bool pr, bool up, size_t &smem) {
    double best = 0.0;
    for (int K : {8, 6, 4, 2}) {
        const int H = K + 1;
        for (int gz = 1; gz <= std::min(blocks, p.n[2]); ++gz)
            for (int gy = 1; gy <= std::min(blocks / gz, p.n[1]); ++gy) {
                const int g[3] = {std::min(blocks / (gz * gy), p.n[0]), gy, gz};
                int wn[3];
                for (int k = 0; k < 3; ++k) {
                    wn[k] = std::min((p.n[k] + g[k] - 1) / g[k] + 2 * H, p.n[k] + 2);
                    if (k == 0) wn[k] += 1;  // the origin rounded down to even
                }
                const size_t need = volume_smem(wn, ks, pr, up);
                if (need > (size_t)SMEM_MAX) continue;
                const int hw = (wn[0] + 1) / 2, rows = wn[1] * wn[2];
                const double updates = (double)rows * hw / 32.0;
                const double half = 300.0 + 30.0 * updates;
                const bool alone = g[0] * g[1] * g[2] == 1;
                const double cost = ((alone ? 1000.0 : MEET_CYCLES) + 10.0 * updates + K * half) / (K / 2);
                if (best == 0.0 || cost < best) {
                    best = cost;
                    for (int k = 0; k < 3; ++k) p.g[k] = g[k];
                    p.k = K;
                    p.most = rows * hw;
                    p.nblocks = g[0] * g[1] * g[2];
                    smem = need;
                }
            }
    }
    return best;
}

typedef void (*Resident)(Args);

template <bool RES>
Resident volume_of(int per) {
    switch (per) {
    case 0:
    case 1: return k_relax64_volume<RES, 1>;
    case 2: return k_relax64_volume<RES, 2>;
    case 3: return k_relax64_volume<RES, 3>;
    case 4: return k_relax64_volume<RES, 4>;
    default: return k_relax64_volume<RES, 0>;
    }
}

template <bool RES, bool GEN>
Resident plane_of(const Shape &sh) {
    if (sh.G == 16) return k_relax64_plane<16, 2, RES, GEN>;
    return sh.R == 2   ? k_relax64_plane<32, 2, RES, GEN>
           : sh.R == 4 ? k_relax64_plane<32, 4, RES, GEN>
                       : k_relax64_plane<32, 8, RES, GEN>;
}

}  // namespace

namespace cw {

// What a field keeps for its resident solves: the second buffer of the
// exchange, the tilings of its histories and the words they meet on.
struct Resident64 {
    double *other = nullptr;
    size_t other_size = 0;         // its numbers, and those the tilings need
    size_t other_need = 0;
    Part *parts = nullptr;
    uint32_t *words = nullptr;     // arrivals, whether a meeting failed, then the slots
    std::vector<Part> host;
    std::vector<Span> spans;       // what the tilings were made for
    const void *coef[3] = {};
    int nsm = 0;
    bool served = false;
    Resident kern[2] = {};         // by the stop: the largest change, the residual
    int threads = RT;
    size_t smem = 0;
};

void resident64_release(cw_field_s *f) {
    Resident64 *r = f->resident;
    if (!r) return;
    dfree(r->other);
    dfree(r->parts);
    dfree(r->words);
    delete r;
    f->resident = nullptr;
}

static bool same_spans(const std::vector<Span> &a, const std::vector<Span> &b) {
    if (a.size() != b.size()) return false;
    for (size_t k = 0; k < a.size(); ++k)
        if (a[k].found != b[k].found || a[k].x0 != b[k].x0 || a[k].x1 != b[k].x1 || a[k].y0 != b[k].y0 ||
            a[k].y1 != b[k].y1 || a[k].z0 != b[k].z0 || a[k].z1 != b[k].z1)
            return false;
    return true;
}

// The tilings for the field's spans and arrays: every history's blocks
// resident at once, one to an SM, shared out by the histories' free spans.
static int resident64_plan(cw_field_s *f, Resident64 *r, const FieldView &fv, const std::vector<Span> &spans) {
    const void *coef[3] = {fv.ks, fv.pr, fv.up};
    if (std::equal(coef, coef + 3, r->coef) && same_spans(r->spans, spans)) return CW_OK;
    r->served = false;
    r->spans = spans;
    std::copy(coef, coef + 3, r->coef);
    r->host.clear();
    int64_t all = 0;
    int live = 0;
    bool volume = false, border = false;
    for (uint32_t k = 0; k < f->g.nh; ++k) {
        volume = volume || f->g.d[k] > 1;
        if (!spans[k].found) continue;
        const Span &s = spans[k];
        all += (int64_t)(s.x1 - s.x0 + 1) * (s.y1 - s.y0 + 1) * (s.z1 - s.z0 + 1);
        border = border || s.x0 == 0 || s.y0 == 0 || s.x1 + 1 == f->g.w[k] || s.y1 + 1 == f->g.h[k];
        ++live;
    }
    if (live == 0 || live > r->nsm) return CW_OK;
    int64_t rows = 0;  // planes: a window's rows
    // a block for each history, the others by size
    std::vector<Part> parts;
    std::vector<int> blocks;
    for (uint32_t k = 0; k < f->g.nh; ++k) {
        const Span &s = spans[k];
        if (!s.found) continue;
        Part p{};
        p.h = (int)k;
        p.lo[0] = s.x0; p.lo[1] = s.y0; p.lo[2] = s.z0;
        p.n[0] = s.x1 - s.x0 + 1; p.n[1] = s.y1 - s.y0 + 1; p.n[2] = s.z1 - s.z0 + 1;
        parts.push_back(p);
        blocks.push_back(1 + (int)((double)(r->nsm - live) * ((double)p.n[0] * p.n[1] * p.n[2]) / (double)all));
    }
    if (volume) {
        int most = 0;
        r->smem = 0;
        r->threads = RT;
        for (size_t k = 0; k < parts.size(); ++k) {
            size_t smem = 0;
            if (plan_volume(parts[k], blocks[k], fv.ks, fv.pr, fv.up, smem) == 0.0) return CW_OK;
            r->smem = std::max(r->smem, smem);
            most = std::max(most, parts[k].most);
        }
        const int per = (most + RT - 1) / RT;
        r->kern[0] = volume_of<false>(per);
        r->kern[1] = volume_of<true>(per);
    } else {
        const bool gen = fv.ks || fv.pr || border;
        std::vector<Part> best;
        double least = 0.0;
        Shape with = SHAPES[0];
        for (const Shape &sh : SHAPES) {
            if (plane_smem(sh, gen, fv.pr, fv.up) > (size_t)SMEM_MAX) continue;
            std::vector<Part> tried = parts;
            double worst = 0.0;  // the slowest history's
            bool fits = true;
            for (size_t k = 0; k < tried.size() && fits; ++k) {
                const double c = plan_plane(tried[k], blocks[k], sh, gen);
                fits = c > 0.0;
                worst = std::max(worst, c);
            }
            if (!fits || (!best.empty() && worst >= least)) continue;
            best = tried;
            least = worst;
            with = sh;
        }
        if (best.empty()) return CW_OK;
        parts = best;
        rows = with.R * (with.threads / with.G);
        r->threads = with.threads;
        r->smem = plane_smem(with, gen, fv.pr, fv.up);
        r->kern[0] = gen ? plane_of<false, true>(with) : plane_of<false, false>(with);
        r->kern[1] = gen ? plane_of<true, true>(with) : plane_of<true, false>(with);
    }
    int first = 0;
    r->other_need = 0;
    for (Part &p : parts) {
        p.first = first;
        first += p.nblocks;
        // a volume's free slices, a plane's rows from the first of a window to the
        // last (`rows` of them below the window's first)
        const int64_t w = f->g.w[p.h], h = f->g.h[p.h];
        int64_t from, to;
        if (volume) {
            from = (int64_t)p.lo[2] * h * w;
            to = (int64_t)(p.lo[2] + p.n[2]) * h * w;
        } else {
            from = std::max(p.lo[1] - 2, 0) * w;
            to = std::min<int64_t>(p.lo[1] + p.n[1] + rows, h) * w;
        }
        p.shift = f->g.off[p.h] + from - (int64_t)r->other_need;
        r->other_need += (size_t)(to - from);
    }
    r->host = parts;
    if (!r->parts && cudaMalloc((void **)&r->parts, sizeof(Part) * f->g.nh) != cudaSuccess) {
        r->parts = nullptr;
        (void)cudaGetLastError();
        r->spans.clear();  // (tried again by the next solve)
        return CW_OK;
    }
    CW_CUDA(cudaMemcpyAsync(r->parts, r->host.data(), sizeof(Part) * r->host.size(), cudaMemcpyHostToDevice, stream()));
    r->served = true;
    return CW_OK;
}

// The FP64 relax on chip, where every history's tiles fit the device at once
// (*served false: they do not, nothing has run).  hs: the histories' states as
// uploaded to d_st; on return what the solve left.
int relax64_resident(cw_field_s *f, const cw_relax_opts &o, const std::vector<Span> &spans, RelaxState *d_st,
                     std::vector<RelaxState> &hs, bool *served) {
    *served = false;
    const uint32_t nh = f->g.nh;
    if (!f->resident) {
        Resident64 *r = new Resident64();
        int dev = 0, coop = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
        cudaDeviceGetAttribute(&r->nsm, cudaDevAttrMultiProcessorCount, dev);
        if (!coop) r->nsm = 0;
        f->resident = r;
    }
    Resident64 *r = f->resident;
    const FieldView fv = view(f);
    int rc = resident64_plan(f, r, fv, spans);
    if (rc != CW_OK || !r->served) return rc;
    const size_t slots = ((size_t)nh + 2) & ~(size_t)1;  // (64-bit words)
    const size_t words = slots + 2 * (size_t)nh * 3 * SLOTS;
    // a device without room for the scratch serves the solve by launches
    if (r->other_need > r->other_size) {
        dfree(r->other);
        r->other_size = 0;
        if (cudaMalloc((void **)&r->other, sizeof(double) * r->other_need) != cudaSuccess) {
            r->other = nullptr;
            (void)cudaGetLastError();
            return CW_OK;
        }
        r->other_size = r->other_need;
    }
    if (!r->words && cudaMalloc((void **)&r->words, sizeof(uint32_t) * words) != cudaSuccess) {
        r->words = nullptr;
        (void)cudaGetLastError();
        return CW_OK;
    }
    const bool res = o.stop == CW_STOP_RESIDUAL;
    const Resident kern = r->kern[res ? 1 : 0];
    CW_CUDA(cudaFuncSetAttribute((const void *)kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_MAX));
    Args a{};
    a.fv = fv;
    a.other = r->other;
    a.parts = r->parts;
    a.nparts = (int)r->host.size();
    a.st = d_st;
    a.arrivals = r->words;
    a.failed = r->words + nh;
    a.slots = (unsigned long long *)(r->words + slots);
    a.wait_ns = test_faults().wait_ns ? test_faults().wait_ns : WAIT_NS;
    a.withhold = test_faults().withhold_block;
    const Part &last = r->host.back();
    void *args[] = {&a};
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.gridDim = dim3((unsigned)(last.first + last.nblocks));
    cfg.blockDim = dim3((unsigned)r->threads);
    cfg.dynamicSmemBytes = r->smem;
    cfg.stream = stream();
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    *served = true;
    for (int64_t taken = 0; taken < o.max_sweeps; taken += a.max_sweeps) {
        if (taken > 0) {
            // the running histories' residual maximum starts again
            for (RelaxState &s : hs)
                if (!s.done) s.resid = 0ull;
            CW_CUDA(cudaMemcpyAsync(d_st, hs.data(), sizeof(RelaxState) * nh, cudaMemcpyHostToDevice, stream()));
        }
        a.max_sweeps = std::min<long long>(LAUNCH_SWEEPS, o.max_sweeps - taken);
        CW_CUDA(cudaMemsetAsync(r->words, 0, sizeof(uint32_t) * words, stream()));
        const cudaError_t launched = cudaLaunchKernelExC(&cfg, (const void *)kern, args);
        if (launched == cudaErrorCooperativeLaunchTooLarge && taken == 0) {
            // fewer SMs for this process than the device has: by launches
            (void)cudaGetLastError();
            *served = false;
            return CW_OK;
        }
        if (launched != cudaSuccess) return cuda_fail(launched, "cooperative launch");
        count_launch(1);
        uint32_t failed = 0;
        CW_CUDA(cudaMemcpyAsync(hs.data(), d_st, sizeof(RelaxState) * nh, cudaMemcpyDeviceToHost, stream()));
        CW_CUDA(cudaMemcpyAsync(&failed, a.failed, sizeof failed, cudaMemcpyDeviceToHost, stream()));
        CW_CUDA(cudaStreamSynchronize(stream()));
        if (failed) return fail(CW_ERR_TIMEOUT, "a block of the FP64 relax waited too long for its history's others");
        bool all = true;
        for (const RelaxState &s : hs) all = all && s.done;
        if (all) break;
    }
    if (!res)
        for (RelaxState &s : hs) s.last_resid = __builtin_bit_cast(double, (uint64_t)s.resid);
    return CW_OK;
}

}  // namespace cw
