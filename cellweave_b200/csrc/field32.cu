// FP32 red-black SOR on the correction equation A d = r of the
// defect-correction solve (see field.cu).  Built with fused multiply-add:
// this is the fast path, and its error is removed by the FP64 residual and
// correction steps.  The coefficients come with the relaxation factor folded
// in (field.cu writes them): b = omega r / den and a = omega D / den, so one
// update is d' = (1 - omega) d + a (sum of the four neighbours) + b, two
// fused multiply-adds after the neighbour sum.
//
// Temporal blocking.  A flat history is cut into windows; a block takes a
// window and runs DEPTH half-sweeps on it before writing its interior back to
// the other buffer.  Every window pixel is updated at every half-sweep, its
// missing neighbours read as zero; the error this makes at a window edge that
// lies inside the history moves in by one ring per half-sweep, so after DEPTH
// of them every pixel at least DEPTH from such an edge is exactly what DEPTH
// global half-sweeps give.  A window edge on or beyond the history's border
// makes no error (outside pixels are zero there too), so the interior reaches
// that border.  The correction crosses HBM once per DEPTH half-sweeps.
//
// The wide kernel (rows 16-byte aligned in every history, the campaign's
// case): 128 x 64 windows, a warp per 16 rows, a lane per 4 consecutive
// columns held as float4 registers (two pixels of each colour per row, one
// warp shuffle per two updates; 244 registers a thread, no spills).  Blocks
// are persistent, two per SM; while a block sweeps one window in registers,
// the TMA engine brings the next window's correction and coefficients into
// shared memory (one mbarrier, 96 KB), so the HBM reads overlap the sweeps.
// Windows start at x = k (128 - 2 DEPTH), a multiple of 4 floats as TMA needs,
// and at y = k (64 - 2 DEPTH).
//
// What bounds it: at depth 8 the four sweeps' own instructions, not HBM (54 us
// of traffic a launch on 64 histories of up to 1024^2, 22.3 M pixels), and next to
// them what a window costs besides: the published rows, the barriers, the
// look-up.  Sixteen rows a warp instead of eight halve the published rows and
// the warps at a barrier per update and let two half-sweeps run unrolled;
// listing 32 windows at a time takes three dependent reads off every window;
// launches that overlap their beginnings take the empty tail of one and the
// set-up of the next off the line.  Together, depth 8, a launch: 92.3 -> 66.4 us
// on that field (62.7 in 128 x 128 windows), 22.9 -> 16.2 on one 2048^2 plane,
// 10.5 -> 7.6 on 1024^2.  Tried and slower: waiting for the neighbours' rows a
// half-sweep later by an mbarrier of arrivals (76.3 against 70.3 without it).
//
// The narrow kernel (any width): 64 x 64 windows, a lane per column pair,
// plain loads, one window per block.  Its launches, and the volumes', overlap
// too: 2.56 -> 2.23 ms the relax of a 1023 x 769 sheet.  Its last launch adds the
// correction as the others' do (two passes of the update, a colour each, took 12
// us apiece where one residual takes 11): 2.23 -> 2.14 ms.
//
// Between warps, each warp publishes its top and bottom rows in shared memory
// after every half-sweep (double-buffered, so one barrier per half-sweep).

#include <mutex>

#include "cw_internal.cuh"
#include "field_kernels.cuh"
#include "tma.cuh"

namespace cw {
namespace {

// ------------------------------------------------------------------ narrow windows

constexpr int WIN = 64;            // window side
constexpr int WARPS = 8;           // warps per block
constexpr int ROWS = WIN / WARPS;  // window rows per warp

// One half-sweep of colour C over the thread's rows (C known at compile
// time: the colour of each row's pixels is then fixed and no branch is left).
// ab/be: the rows just above and below this warp's, from the neighbours.
template <int C>
__device__ __forceinline__ void half_sweep(float (&d0)[ROWS], float (&d1)[ROWS], const float (&r0)[ROWS],
                                           const float (&r1)[ROWS], const float (&i0)[ROWS],
                                           const float (&i1)[ROWS], float ab0, float ab1, float be0, float be1,
                                           float lm, float rm, float omc) {
#pragma unroll
    for (int j = 0; j < ROWS; ++j) {
        if (((C + j) & 1) == 0) {  // the even column of the pair
            const float left = __shfl_up_sync(0xffffffffu, d1[j], 1);
            const float up = j > 0 ? d0[j - 1] : ab0, down = j < ROWS - 1 ? d0[j + 1] : be0;
            d0[j] = fmaf(i0[j], fmaf(lm, left, d1[j]) + (up + down), fmaf(omc, d0[j], r0[j]));
        } else {  // the odd column
            const float right = __shfl_down_sync(0xffffffffu, d0[j], 1);
            const float up = j > 0 ? d1[j - 1] : ab1, down = j < ROWS - 1 ? d1[j + 1] : be1;
            d1[j] = fmaf(i1[j], fmaf(rm, right, d0[j]) + (up + down), fmaf(omc, d1[j], r1[j]));
        }
    }
}

// (src not restricted: an overlapped launch's blocks are there while the launch
// before still writes it, which the read-only path does not allow for)
template <int DEPTH>
__global__ void __launch_bounds__(32 * WARPS) k_sor32_tb(const float *src, float *__restrict__ dst,
                                                         const float *__restrict__ rhs, const float *__restrict__ inv,
                                                         const int4 *__restrict__ dims,
                                                         const int64_t *__restrict__ off,
                                                         const int32_t *__restrict__ blk, int nh,
                                                         const float *__restrict__ omega, const int32_t *done,
                                                         int done_stride, int nhalf, int zero_start,
                                                         double *__restrict__ apply_c,
                                                         const uint8_t *__restrict__ held, int floor) {
    constexpr int IN = WIN - 2 * DEPTH;  // interior side
    // edge rows each warp publishes, double-buffered by half-sweep parity:
    // [buffer][warp][0 top, 1 bottom][column]
    __shared__ float edge[2][WARPS][2][WIN];
    __shared__ int s_h;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) s_h = plan_history(blk, nh, blockIdx.x);
    __syncthreads();
    const int h = s_h;
    const bool idle = done[(int64_t)h * done_stride];
    await_previous();
    let_next_begin();
    if (idle) return;
    const int4 dm = dims[h];
    const int ntx = (dm.x + IN - 1) / IN;
    const int t = blockIdx.x - blk[h];
    const int gx0 = (t % ntx) * IN - DEPTH, gy0 = (t / ntx) * IN - DEPTH;
    const int64_t base = off[h];
    const float omc = 1.f - omega[h];
    // the lanes at the window's sides have no neighbour across it (a zero);
    // the shuffle's own value, finite, is multiplied by zero instead
    const float lm = lane == 0 ? 0.f : 1.f, rm = lane == 31 ? 0.f : 1.f;
    const int gx = gx0 + 2 * lane;
    const bool in0 = gx >= 0 && gx < dm.x, in1 = gx + 1 >= 0 && gx + 1 < dm.x;
    float d0[ROWS], d1[ROWS], r0[ROWS], r1[ROWS], i0[ROWS], i1[ROWS];
#pragma unroll
    for (int j = 0; j < ROWS; ++j) {
        const int gy = gy0 + ROWS * warp + j;
        d0[j] = d1[j] = r0[j] = r1[j] = i0[j] = i1[j] = 0.f;
        if (gy >= 0 && gy < dm.y) {
            const int64_t row = base + (int64_t)gy * dm.x + gx;
            if (in0) { d0[j] = zero_start ? 0.f : src[row]; r0[j] = rhs[row]; i0[j] = inv[row]; }
            if (in1) { d1[j] = zero_start ? 0.f : src[row + 1]; r1[j] = rhs[row + 1]; i1[j] = inv[row + 1]; }
        }
    }
    auto publish = [&](int buf) {
        edge[buf][warp][0][2 * lane] = d0[0];
        edge[buf][warp][0][2 * lane + 1] = d1[0];
        edge[buf][warp][1][2 * lane] = d0[ROWS - 1];
        edge[buf][warp][1][2 * lane + 1] = d1[ROWS - 1];
    };
    publish(0);
    __syncthreads();
    // window pixel (ex, ey) has colour (gx0 + gy0 + ex + ey) mod 2, and gx0 + gy0
    // and 8 warp are even: in row j the pixel of colour c is the pair's (c + j) mod 2
    for (int s = 0; s < nhalf; ++s) {
        const int buf = s & 1;
        const float ab0 = warp > 0 ? edge[buf][warp - 1][1][2 * lane] : 0.f;
        const float ab1 = warp > 0 ? edge[buf][warp - 1][1][2 * lane + 1] : 0.f;
        const float be0 = warp < WARPS - 1 ? edge[buf][warp + 1][0][2 * lane] : 0.f;
        const float be1 = warp < WARPS - 1 ? edge[buf][warp + 1][0][2 * lane + 1] : 0.f;
        if ((s & 1) == 0)
            half_sweep<0>(d0, d1, r0, r1, i0, i1, ab0, ab1, be0, be1, lm, rm, omc);
        else
            half_sweep<1>(d0, d1, r0, r1, i0, i1, ab0, ab1, be0, be1, lm, rm, omc);
        // the other buffer was last read before the previous barrier
        publish(buf ^ 1);
        __syncthreads();
    }
    // the interior back to global memory
#pragma unroll
    for (int j = 0; j < ROWS; ++j) {
        const int ey = ROWS * warp + j, gy = gy0 + ey;
        if (ey < DEPTH || ey >= DEPTH + IN || gy >= dm.y) continue;
        const int64_t row = base + (int64_t)gy * dm.x + gx;
        const int ex = 2 * lane;
        const bool out0 = ex >= DEPTH && ex < DEPTH + IN && gx < dm.x;
        const bool out1 = ex + 1 >= DEPTH && ex + 1 < DEPTH + IN && gx + 1 < dm.x;
        if (apply_c) {
            // a solve's last launch: c += d on the free pixels
            if (out0 && !held[row]) {
                const double c = apply_c[row] + (double)d0[j];
                apply_c[row] = floor ? fmax(c, 0.0) : c;
            }
            if (out1 && !held[row + 1]) {
                const double c = apply_c[row + 1] + (double)d1[j];
                apply_c[row + 1] = floor ? fmax(c, 0.0) : c;
            }
            continue;
        }
        if (out0) dst[row] = d0[j];
        if (out1) dst[row + 1] = d1[j];
    }
}

// ------------------------------------------------------------------ wide windows (TMA)

constexpr int WX = 128;              // window columns
constexpr int WROWS = 16;            // rows per warp; a window has WROWS rows per warp of its block
// Two shapes: 128 x 64 windows, two blocks per SM, or 128 x 128 windows, one
// block per SM: a smaller share of the window is halo, 1.31 pixels swept per
// interior pixel at depth 8 against 1.52.
constexpr size_t wide_smem(int warps) {
    return (size_t)3 * WX * WROWS * warps * sizeof(float) + (size_t)2 * (warps + 2) * 2 * (WX / 4) * sizeof(float4);
}

// One half-sweep of colour C over a lane's WROWS rows x 4 columns.  Column c
// of row j has colour (c + j) mod 2 (windows start at even x and y): colour C
// takes columns 0 and 2 of the rows with C + j even, 1 and 3 of the others.
// Every update reads only pixels of the other colour, which this half-sweep
// does not change.
template <int C>
__device__ __forceinline__ void rows4(float4 (&d)[WROWS], const float4 (&a)[WROWS], const float4 (&b)[WROWS],
                                      const float4 ab, const float4 be, float lm, float rm, float omc) {
#pragma unroll
    for (int j0 = 0; j0 < WROWS; j0 += 8) {
        // eight rows' across-lane neighbours first: they are of the other
        // colour, and their latency then overlaps
        float nb[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const int j = j0 + q;
            nb[q] = ((C + j) & 1) == 0 ? __shfl_up_sync(0xffffffffu, d[j].w, 1)
                                       : __shfl_down_sync(0xffffffffu, d[j].x, 1);
        }
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const int j = j0 + q;
            const float4 up = j > 0 ? d[j > 0 ? j - 1 : 0] : ab, dn = j < WROWS - 1 ? d[j < WROWS - 1 ? j + 1 : j] : be;
            if (((C + j) & 1) == 0) {
                const float s0 = fmaf(lm, nb[q], d[j].y) + (up.x + dn.x);
                const float s2 = (d[j].y + d[j].w) + (up.z + dn.z);
                d[j].x = fmaf(a[j].x, s0, fmaf(omc, d[j].x, b[j].x));
                d[j].z = fmaf(a[j].z, s2, fmaf(omc, d[j].z, b[j].z));
            } else {
                const float s1 = (d[j].x + d[j].z) + (up.y + dn.y);
                const float s3 = fmaf(rm, nb[q], d[j].z) + (up.w + dn.w);
                d[j].y = fmaf(a[j].y, s1, fmaf(omc, d[j].y, b[j].y));
                d[j].w = fmaf(a[j].w, s3, fmaf(omc, d[j].w, b[j].w));
            }
        }
    }
}

// What a block needs of a window.  A block's next 32 are looked up at once, a
// lane each, and the live ones listed in shared memory: looking up one at each
// window's turn (its record, whether its history has settled, then the
// history's scalars: three reads in turn by one thread, the block waiting) took
// a fifth of a window's time.
struct WideTile {
    int4 tl;      // (history, x0, y0, 0)
    int4 dm;      // the history's dimensions
    int64_t off;  // its first pixel
    float omc;    // 1 - omega
};

// maps: 4 per history (d32a, d32b, r32, inv32); src_map picks the buffer
// read (0 or 1), dst is the other.  tiles: (history, x0, y0, 0) per window.
// zero_start: the correction starts at zero (the first launch of a solve):
// it is not read.  apply_c: the last launch of a solve adds its correction to
// the FP64 field (floored at zero when `floor`) instead of writing it to dst.
template <int DEPTH, int WWARPS>
__global__ void __launch_bounds__(32 * WWARPS, WWARPS * WROWS == 64 ? 2 : 1)
    k_sor32_wide(const CUtensorMap *__restrict__ maps, int src_map, float *__restrict__ dst,
                 const int4 *__restrict__ tiles, int ntiles, const int4 *__restrict__ dims,
                 const int64_t *__restrict__ off, const float *__restrict__ omega, const int32_t *done,
                 int done_stride, int nhalf, int zero_start, double *__restrict__ apply_c,
                 int floor, unsigned long long wait_ns, int skip_copies, unsigned long long *corr, int corr_stride,
                 uint32_t *failed) {
    constexpr int WY = WROWS * WWARPS;  // window rows
    constexpr int STAGE = WX * WY;      // floats per array of the staged window
    extern __shared__ __align__(128) float smem[];
    const float4 *sd = (const float4 *)smem, *sb = (const float4 *)(smem + STAGE),
                 *sa = (const float4 *)(smem + 2 * STAGE);
    // [buffer][warp + 1][0 top, 1 bottom][lane], a warp of zeros at either end
    float4 *edge = (float4 *)(smem + 3 * STAGE);
    constexpr int EBUF_ALL = (WWARPS + 2) * 64;
    __shared__ __align__(8) uint64_t bar_word;
    __shared__ WideTile s_tile[32];
    __shared__ int s_tiles, s_from, s_fail;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t bar = sh_addr(&bar_word);
    const uint32_t boxes = zero_start ? 2u : 3u;
    // warp 0: the live ones of this block's windows from `from` on, until there
    // is one or no window is left
    auto look_up = [&](int from) {
        unsigned live = 0;
        for (; live == 0u && from < ntiles; from += 32 * gridDim.x) {
            const int t = from + lane * gridDim.x;
            int4 tl = make_int4(0, 0, 0, 0);
            bool on = t < ntiles;
            if (on) {
                tl = tiles[t];
                on = !done[(int64_t)tl.x * done_stride];
            }
            live = __ballot_sync(0xffffffffu, on);
            if (on) {
                WideTile &w = s_tile[__popc(live & ((1u << lane) - 1u))];
                w.tl = tl;
                w.dm = dims[tl.x];
                w.off = off[tl.x];
                w.omc = 1.f - omega[tl.x];
            }
        }
        if (lane == 0) {
            s_tiles = __popc(live);
            s_from = from;
        }
        __syncwarp();
    };
    // thread 0: start the copies of a listed window
    auto copy = [&](const int4 tl) {
        const CUtensorMap *m = maps + 4 * tl.x;
        mbar_expect_tx(bar, (uint32_t)(boxes * STAGE * sizeof(float)));
        // skip_copies (a failure test): the bytes announced never come,
        // and the wait below runs out
        if (!skip_copies) {
            if (!zero_start) tma_load_2d(smem, m + src_map, bar, tl.y, tl.z);
            tma_load_2d(smem + STAGE, m + 2, bar, tl.y, tl.z);
            tma_load_2d(smem + 2 * STAGE, m + 3, bar, tl.y, tl.z);
        }
    };
    for (int i = threadIdx.x; i < 2 * EBUF_ALL; i += 32 * WWARPS) edge[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (threadIdx.x == 0) {
        mbar_init(bar, 1);
        mbar_init_fence();
        s_fail = 0;
    }
    // (a launch that overlaps another follows a sweep, which does not write
    // what the look-up reads; the buffers wait for that sweep's end)
    if (warp == 0) look_up(blockIdx.x);
    await_previous();
    let_next_begin();
    if (threadIdx.x == 0 && s_tiles > 0) copy(s_tile[0].tl);
    __syncthreads();
    uint32_t parity = 0;
    const float lm = lane == 0 ? 0.f : 1.f, rm = lane == 31 ? 0.f : 1.f;
    const float4 z4 = make_float4(0.f, 0.f, 0.f, 0.f);
    // this lane's published top row in either buffer; the bottom row 32 behind,
    // the warps above and below 64 before and behind
    constexpr int EBUF = EBUF_ALL;
    float4 *const my_edge = edge + (warp + 1) * 64 + lane;
    for (int k = 0; k < s_tiles;) {
        const WideTile info = s_tile[k];
        const bool relist = k + 1 == s_tiles;  // read before warp 0 lists anew
        if (!mbar_wait_bounded(bar, parity, wait_ns)) s_fail = 1;
        float4 d[WROWS], a[WROWS], b[WROWS];
#pragma unroll
        for (int j = 0; j < WROWS; ++j) {
            const int q = (warp * WROWS + j) * 32 + lane;
            d[j] = zero_start ? z4 : sd[q];
            b[j] = sb[q];
            a[j] = sa[q];
        }
        __syncthreads();  // the stage is read: free for the next window
        if (s_fail) {
            // leave no copy in flight into this block's shared memory
            if (threadIdx.x == 0) {
                mbar_wait_bounded(bar, parity, wait_ns);
                atomicExch(failed, 1u);
            }
            return;
        }
        parity ^= 1u;
        // the next window, from the list or a new one
        k = relist ? 0 : k + 1;
        if (warp == 0) {
            if (relist) look_up(s_from);
            if (lane == 0 && s_tiles > 0) {
                // the generic-proxy reads of the stage before the async-proxy writes
                fence_proxy_async_shared();
                copy(s_tile[k].tl);
            }
        }
        const float omc = info.omc;
        my_edge[0] = d[0];
        my_edge[32] = d[WROWS - 1];
        __syncthreads();
        // (a launch's half-sweeps are even in number and begin with the red: two a turn)
        for (int s = 0; s < nhalf; s += 2) {
            rows4<0>(d, a, b, my_edge[-32], my_edge[64], lm, rm, omc);
            // the other buffer was last read before the previous barrier
            my_edge[EBUF] = d[0];
            my_edge[EBUF + 32] = d[WROWS - 1];
            __syncthreads();
            rows4<1>(d, a, b, my_edge[EBUF - 32], my_edge[EBUF + 64], lm, rm, omc);
            if (s + 2 < nhalf) {
                my_edge[0] = d[0];
                my_edge[32] = d[WROWS - 1];
                __syncthreads();
            }
        }
        // the interior back to global memory: the warp's rows inside it (a
        // range uniform over the warp), the lane's columns inside it (all four,
        // none, or a few at a history border that cuts a float4)
        const int x0 = info.tl.y, y0 = info.tl.z;
        const int4 dm = info.dm;
        const int ix0 = x0 == 0 ? 0 : x0 + DEPTH, ix1 = x0 + WX >= dm.x ? dm.x : x0 + WX - DEPTH;
        const int iy0 = y0 == 0 ? 0 : y0 + DEPTH, iy1 = y0 + WY >= dm.y ? dm.y : y0 + WY - DEPTH;
        const int wy = y0 + warp * WROWS;
        const int j0 = max(iy0 - wy, 0), j1 = min(iy1 - wy, WROWS);
        const int gx = x0 + 4 * lane;
        const bool full = gx >= ix0 && gx + 4 <= ix1;
        const bool part = !full && gx + 4 > ix0 && gx < ix1;
        const int64_t first = info.off + (int64_t)wy * dm.x + gx;
        if (apply_c) {
            // c += d on the free pixels (held ones have a = 0 and d = 0 throughout)
            double *row = apply_c + first;
            float most = 0.f;   // the largest |d| the window adds
            double top = 0.0;   // and the largest |c| it leaves
#pragma unroll
            for (int j = 0; j < WROWS; ++j, row += dm.x) {
                if (j < j0 || j >= j1 || !(full || part)) continue;
                const float dv[4] = {d[j].x, d[j].y, d[j].z, d[j].w};
                const float av[4] = {a[j].x, a[j].y, a[j].z, a[j].w};
                if (corr) {
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                        if (full || (gx + e >= ix0 && gx + e < ix1)) most = fmaxf(most, fabsf(dv[e]));
                }
                if (full) {
                    double2 c01 = *(double2 *)row, c23 = *(double2 *)(row + 2);
                    double cv[4] = {c01.x, c01.y, c23.x, c23.y};
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                        if (dv[e] != 0.f || av[e] != 0.f) {
                            cv[e] = cv[e] + (double)dv[e];
                            if (floor) cv[e] = fmax(cv[e], 0.0);
                            top = fmax(top, fabs(cv[e]));
                        }
                    *(double2 *)row = make_double2(cv[0], cv[1]);
                    *(double2 *)(row + 2) = make_double2(cv[2], cv[3]);
                } else {
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                        if (gx + e >= ix0 && gx + e < ix1 && (dv[e] != 0.f || av[e] != 0.f)) {
                            double v = row[e] + (double)dv[e];
                            row[e] = floor ? fmax(v, 0.0) : v;
                            top = fmax(top, fabs(row[e]));
                        }
                }
            }
            if (corr) {
                // one atomic per warp and window
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) most = fmaxf(most, __shfl_xor_sync(0xffffffffu, most, o));
                for (int o = 16; o > 0; o >>= 1) top = fmax(top, __shfl_xor_sync(0xffffffffu, top, o));
                if (lane == 0) {
                    unsigned long long *mine = corr + (int64_t)info.tl.x * corr_stride;
                    if (most > 0.f) atomicMax(mine, (unsigned long long)__double_as_longlong((double)most));
                    if (top > 0.0) atomicMax(mine + 1, (unsigned long long)__double_as_longlong(top));
                }
            }
        } else if (j0 <= 0 && j1 >= WROWS) {
            // every row of the warp (most warps)
            float *row = dst + first;
            if (full) {
#pragma unroll
                for (int j = 0; j < WROWS; ++j, row += dm.x) *(float4 *)row = d[j];
            } else if (part) {
#pragma unroll
                for (int j = 0; j < WROWS; ++j, row += dm.x) {
                    if (gx >= ix0 && gx < ix1) row[0] = d[j].x;
                    if (gx + 1 >= ix0 && gx + 1 < ix1) row[1] = d[j].y;
                    if (gx + 2 >= ix0 && gx + 2 < ix1) row[2] = d[j].z;
                    if (gx + 3 >= ix0 && gx + 3 < ix1) row[3] = d[j].w;
                }
            }
        } else {
            float *row = dst + first;
#pragma unroll
            for (int j = 0; j < WROWS; ++j, row += dm.x) {
                if (j < j0 || j >= j1) continue;
                if (full) {
                    *(float4 *)row = d[j];
                } else if (part) {
                    if (gx >= ix0 && gx < ix1) row[0] = d[j].x;
                    if (gx + 1 >= ix0 && gx + 1 < ix1) row[1] = d[j].y;
                    if (gx + 2 >= ix0 && gx + 2 < ix1) row[2] = d[j].z;
                    if (gx + 3 >= ix0 && gx + 3 < ix1) row[3] = d[j].w;
                }
            }
        }
    }
}

// ------------------------------------------------------------------ volumes

// One half-sweep in place, any depth of lattice (volumes).
__global__ void k_sor32_half(float *__restrict__ dlt, const float *__restrict__ rhs, const float *__restrict__ inv,
                             const int4 *__restrict__ dims, const int64_t *__restrict__ off,
                             const int32_t *__restrict__ blk, int nh, const float *__restrict__ omega,
                             const int32_t *done, int done_stride, int colour) {
    __shared__ int s_h;
    if (threadIdx.x == 0) s_h = plan_history(blk, nh, blockIdx.x);
    __syncthreads();
    const int h = s_h;
    if (done[(int64_t)h * done_stride]) return;
    const int4 dm = dims[h];
    const int hw = (dm.x + 1) >> 1;
    int64_t k = (int64_t)(blockIdx.x - blk[h]) * blockDim.x + threadIdx.x;
    int64_t rows = (int64_t)dm.y * dm.z;
    if (k >= rows * hw) return;
    int64_t row = k / hw;
    int y = (int)(row % dm.y), z = (int)(row / dm.y);
    int x = ((colour - y - z) & 1) + 2 * (int)(k - row * hw);
    if (x >= dm.x) return;
    int64_t w = dm.x, slice = (int64_t)dm.x * dm.y;
    int64_t i = off[h] + row * w + x;
    // (x pair) + (y pair) [+ (z pair)]: in 2D the windowed kernels' order
    const float xm = x > 0 ? dlt[i - 1] : 0.f, xp = x + 1 < dm.x ? dlt[i + 1] : 0.f;
    const float ym = y > 0 ? dlt[i - w] : 0.f, yp = y + 1 < dm.y ? dlt[i + w] : 0.f;
    float sum = (xm + xp) + (ym + yp);
    if (dm.z > 1) sum += (z > 0 ? dlt[i - slice] : 0.f) + (z + 1 < dm.z ? dlt[i + slice] : 0.f);
    dlt[i] = fmaf(inv[i], sum, fmaf(1.f - omega[h], dlt[i], rhs[i]));
}

// ------------------------------------------------------------------ volumes, blocked

// Temporal blocking in a volume (2.5-D: tiles across x and y marched along
// z).  A block takes a VX x 2 NW tile of a history's columns over a chunk of
// its slices [z0, z1) and runs S <= VD half-sweeps on it in one pass along z:
// at step t, stage s (the s-th half-sweep) updates slice t - (s - 1), the
// pixels of that half-sweep's colour.  A thread owns a pair of columns in two
// rows and keeps the slices in use, t - VD to t + 1, and their coefficients in
// registers, so that a pixel's neighbours along z are its own (slice p + 1 has
// had stage s - 1 in the same step, slice p - 1 a step ago), along x a shuffle,
// along y the thread's other row or the neighbouring warp's: as loaded for the
// first stage, then published in shared memory after each stage for the next
// step.  One barrier a step.  The slices' slots and the colour of each row's
// pixel are known at compile time (steps unrolled over the slots, an even
// number; tiles start at even x, y and z): at step K of the unrolled loop every
// stage updates column (row + K) mod 2 of the pair.
//
// Slices come into a ring in shared memory by asynchronous copies of ALIGN
// bytes (16, 8 or 4, as the histories' rows allow), four slices ahead of the
// one a step reads: with the slices loaded into registers two ahead, waiting
// for them was the first stall.
//
// The tile's halo is VD pixels across x and y and VD slices along z beyond the
// chunk; what lies outside the history or beyond the loaded slices has zero
// coefficients and stays zero: exact at the history's border, and an error
// that moves in one ring per half-sweep inside it, so every pixel VD or more
// from such an edge equals S in-place half-sweeps of the whole history (as
// k_sor32_half gives them, to the bit: the same sums in the same order).
//
// Measured on an oxygen field of 256^3 voxels (16-byte copies): 140 -> 39 us a
// sweep against the kernel before, which kept the slices in shared memory, two
// steps apart, and took 223 thread instructions an update (20 now); its HBM
// floor at two sweeps a launch is 20 us, and the shared-memory pipe is busy 75 %
// of the time.  255^3 (4-byte copies) 140 -> 56, 181^3 53 -> 26, 97^3 22.7 ->
// 10.4, 96^3 21.7 -> 7.4.
constexpr int VX = 64;  // tile columns: 32 lanes x 2
constexpr int VD = 4;   // half-sweeps a launch at most
constexpr int VSLOTS = VD + 2;  // slices in registers, and in the ring

constexpr size_t vol_smem(int nw) {
    return sizeof(float) * ((size_t)VSLOTS * 3 * VX * 2 * nw + 2 * (VD - 1) * (nw + 2) * 64);
}

// ALIGN bytes into shared memory at `to`; zeros where the chunk is not live.
template <int ALIGN>
__device__ __forceinline__ void copy_async(uint32_t to, const float *from, bool live) {
    const int bytes = live ? ALIGN : 0;
    if (ALIGN == 16)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(to), "l"(from), "r"(bytes) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(to), "l"(from), "n"(ALIGN), "r"(bytes)
                     : "memory");
}

// What a launch is, known at compile time: VD half-sweeps in the middle of a
// correction, its first launch (from zero) or its last (the correction added to
// the field); ANY: told at run time, for a launch of fewer half-sweeps.  Without
// the other cases' code the unrolled steps fit the instruction cache (89 -> 62
// us a sweep of 256^3 before the ring; the first and last launch of a
// correction, both ANY before: 115 us on average over a step's, now 51 and 132,
// where the middle ones take 53; launches that find the field settled among them).
enum VolKind { VOL_ANY, VOL_MIDDLE, VOL_FIRST, VOL_LAST };
template <int NW, int ALIGN, int KIND>
__global__ void __launch_bounds__(32 * NW, NW == 16 ? 1 : 2)
    k_sor32_vol(const float *__restrict__ src, float *__restrict__ dst, const float *__restrict__ rhs,
                const float *__restrict__ inv, const int4 *__restrict__ dims, const int64_t *__restrict__ off,
                const int4 *__restrict__ tiles, int vz, const float *__restrict__ omega, const int32_t *done,
                int done_stride, int nhalf, int zero_start, double *__restrict__ apply_c, int floor) {
    constexpr int D = VD, NS = VSLOTS;
    static_assert(NS % 2 == 0, "the steps' parity repeats with the slots");
    constexpr int VY = 2 * NW, ARR = VX * VY, SLICE = 3 * ARR;
    extern __shared__ __align__(16) float vsm[];
    // the ring: [slot][correction, b, a][row][column]; then the published rows:
    // [step parity][stage 1 .. D - 1][warp + 1][row][lane], a warp of zeros at either end
    float *const edge = vsm + NS * SLICE;
    constexpr int EWARP = 64, ESTAGE = (NW + 2) * EWARP, EBUF = (D - 1) * ESTAGE;
    const int4 tl = tiles[blockIdx.x];
    const int h = tl.x;
    const bool idle = done[(int64_t)h * done_stride];
    await_previous();
    let_next_begin();
    if (idle) return;
    const int4 dm = dims[h];
    const int x0 = tl.y, y0 = tl.z, z0 = tl.w;
    const int z1 = min(z0 + vz, dm.z);
    const int zlo = max(z0 - D, 0), zhi = min(z1 + D, dm.z);
    const int S = KIND != VOL_ANY ? D : nhalf;
    if (KIND != VOL_ANY) zero_start = KIND == VOL_FIRST;
    if (KIND == VOL_MIDDLE || KIND == VOL_FIRST) apply_c = nullptr;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int gx = x0 + 2 * lane, gy = y0 + 2 * warp;
    // offsets inside the history in 32 bits (a history holds fewer than 2^31
    // pixels), its arrays from their first pixel
    const int plane = dm.x * dm.y;
    const int64_t base = off[h];
    const float *const from[3] = {src + base, rhs + base, inv + base};
    float *hdst = dst + base;
    double *hc = KIND == VOL_LAST || apply_c ? apply_c + base : nullptr;
    const float omc = 1.f - omega[h];
    const float lm = lane == 0 ? 0.f : 1.f, rm = lane == 31 ? 0.f : 1.f;
    // the output interior of the tile (a window edge on the history's border makes no error)
    const int ix0 = x0 == 0 ? 0 : x0 + D, ix1 = x0 + VX >= dm.x ? dm.x : x0 + VX - D;
    const int iy0 = y0 == 0 ? 0 : y0 + D, iy1 = y0 + VY >= dm.y ? dm.y : y0 + VY - D;
    bool out0[2], out1[2];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        const bool oy = gy + j >= iy0 && gy + j < iy1;
        out0[j] = oy && gx >= ix0 && gx < ix1;
        out1[j] = oy && gx + 1 >= ix0 && gx + 1 < ix1;
    }
    // the chunks of a slice this thread copies of each array: 16 / ALIGN of them
    constexpr int CH = 16 / ALIGN, PER_ROW = VX * 4 / ALIGN, RSTEP = 32 * NW / PER_ROW;
    const int crow = threadIdx.x / PER_ROW, ccol = threadIdx.x % PER_ROW * (ALIGN / 4);
    const uint32_t ring0 = sh_addr(vsm) + 4u * (uint32_t)(crow * VX + ccol);
    const int cfirst = (y0 + crow) * dm.x + x0 + ccol;
    // slice z into slot k of the ring
    auto fetch = [&](int z, int k) {
#pragma unroll
        for (int q = 0; q < CH; ++q) {
            const bool live = x0 + ccol < dm.x && z < zhi && y0 + crow + q * RSTEP < dm.y;
            const int i = live ? z * plane + cfirst + q * RSTEP * dm.x : 0;
#pragma unroll
            for (int m = 0; m < 3; ++m)
                copy_async<ALIGN>(ring0 + 4u * (uint32_t)(k * SLICE + m * ARR + q * RSTEP * VX), from[m] + i,
                                  live && !(m == 0 && zero_start));
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    for (int i = threadIdx.x; i < 2 * EBUF; i += 32 * NW) edge[i] = 0.f;
#pragma unroll
    for (int k = 0; k < NS - 1; ++k) fetch(zlo + k, k);
    float2 v[NS][2], b[NS][2], a[NS][2];
#pragma unroll
    for (int k = 0; k < NS; ++k)
#pragma unroll
        for (int j = 0; j < 2; ++j) v[k][j] = b[k][j] = a[k][j] = make_float2(0.f, 0.f);
    const float *const mine = vsm + 2 * warp * VX + 2 * lane;
    float *const my_edge = edge + (warp + 1) * EWARP + lane;
    auto take = [&](int k, float2 (&V)[2], float2 (&B)[2], float2 (&A)[2]) {
        const float *p = mine + k * SLICE;
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            V[j] = *(const float2 *)(p + j * VX);
            B[j] = *(const float2 *)(p + ARR + j * VX);
            A[j] = *(const float2 *)(p + 2 * ARR + j * VX);
        }
    };
    asm volatile("cp.async.wait_group %0;" ::"n"(NS - 2) : "memory");
    __syncthreads();
    take(0, v[0], b[0], a[0]);
    const int tend = zhi - 1 + (S - 1);
    for (int t0 = zlo; t0 <= tend; t0 += NS) {
#pragma unroll
        for (int K = 0; K < NS; ++K) {
            const int t = t0 + K;
            if (t > tend) break;  // the same for the whole block
            // slice t + 1 has landed for every thread; slice t - 1 has been read
            // by all, its slot takes slice t + NS - 1
            asm volatile("cp.async.wait_group %0;" ::"n"(NS - 3) : "memory");
            __syncthreads();
            fetch(t + NS - 1, (K + NS - 1) % NS);
            // the field's slice that leaves D - 1 steps from now, into L2
            if (KIND == VOL_LAST && t >= z0 && t < z1) {
#pragma unroll
                for (int j = 0; j < 2; ++j)
                    if (out0[j]) asm volatile("prefetch.global.L2 [%0];" ::"l"(hc + t * plane + (gy + j) * dm.x + gx));
            }
            take((K + 1) % NS, v[(K + 1) % NS], b[(K + 1) % NS], a[(K + 1) % NS]);
            // the pixels above and below as loaded, for the first stage
            float above0 = 0.f, below0 = 0.f;
            if (warp > 0) above0 = mine[K * SLICE - VX + (K & 1)];
            if (warp < NW - 1) below0 = mine[K * SLICE + 2 * VX + ((K + 1) & 1)];
            const float *ein = my_edge + (K & 1) * EBUF;
            float *eout = my_edge + ((K + 1) & 1) * EBUF;
#pragma unroll
            for (int s = 1; s <= D; ++s) {
                if (s > S) break;
                const int p = (K - (s - 1) + NS) % NS, pm = (p + NS - 1) % NS, pp = (p + 1) % NS;
                // the across-lane neighbours of both rows first
                float side[2], next[2];
#pragma unroll
                for (int j = 0; j < 2; ++j)
                    side[j] = ((j + K) & 1) == 0 ? __shfl_up_sync(0xffffffffu, v[p][j].y, 1)
                                                 : __shfl_down_sync(0xffffffffu, v[p][j].x, 1);
                const float above = s == 1 ? above0 : ein[(s - 2) * ESTAGE - EWARP + 32];
                const float below = s == 1 ? below0 : ein[(s - 2) * ESTAGE + EWARP];
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    // k_sor32_half's sums, in its order
                    const float2 other = v[p][1 - j];
                    if (((j + K) & 1) == 0) {
                        const float ym = j == 0 ? above : other.x, yp = j == 0 ? other.x : below;
                        float sum = fmaf(lm, side[j], v[p][j].y) + (ym + yp);
                        sum += v[pm][j].x + v[pp][j].x;
                        next[j] = fmaf(a[p][j].x, sum, fmaf(omc, v[p][j].x, b[p][j].x));
                    } else {
                        const float ym = j == 0 ? above : other.y, yp = j == 0 ? other.y : below;
                        float sum = fmaf(rm, side[j], v[p][j].x) + (ym + yp);
                        sum += v[pm][j].y + v[pp][j].y;
                        next[j] = fmaf(a[p][j].y, sum, fmaf(omc, v[p][j].y, b[p][j].y));
                    }
                }
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    if (((j + K) & 1) == 0) v[p][j].x = next[j];
                    else v[p][j].y = next[j];
                    if (s < D) eout[(s - 1) * ESTAGE + 32 * j] = next[j];
                }
                // slice t - (S - 1) has had every half-sweep: its interior out
                const int pf = t - (s - 1);
                if (s == S && pf >= z0 && pf < z1) {
#pragma unroll
                    for (int j = 0; j < 2; ++j) {
                        const int i = pf * plane + (gy + j) * dm.x + gx;
                        const float2 q = v[p][j];
                        if (KIND == VOL_LAST || hc) {
                            // the last launch of a correction: c += d on the free
                            // pixels (a held pixel has a = 0 and d = 0 throughout),
                            // floored as the reference's update is (pde.rs:395)
                            if (ALIGN >= 8 && out0[j] && out1[j]) {
                                double2 c = *(const double2 *)(hc + i);
                                if (q.x != 0.f || a[p][j].x != 0.f) {
                                    c.x = c.x + (double)q.x;
                                    if (floor) c.x = fmax(c.x, 0.0);
                                }
                                if (q.y != 0.f || a[p][j].y != 0.f) {
                                    c.y = c.y + (double)q.y;
                                    if (floor) c.y = fmax(c.y, 0.0);
                                }
                                *(double2 *)(hc + i) = c;
                                continue;
                            }
                            if (out0[j] && (q.x != 0.f || a[p][j].x != 0.f)) {
                                const double c = hc[i] + (double)q.x;
                                hc[i] = floor ? fmax(c, 0.0) : c;
                            }
                            if (out1[j] && (q.y != 0.f || a[p][j].y != 0.f)) {
                                const double c = hc[i + 1] + (double)q.y;
                                hc[i + 1] = floor ? fmax(c, 0.0) : c;
                            }
                        } else if (ALIGN >= 8 && out0[j] && out1[j]) {
                            *(float2 *)(hdst + i) = q;
                        } else {
                            if (out0[j]) hdst[i] = q.x;
                            if (out1[j]) hdst[i + 1] = q.y;
                        }
                    }
                }
            }
        }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
}

typedef void (*TbKernel)(const float *, float *, const float *, const float *, const int4 *, const int64_t *,
                         const int32_t *, int, const float *, const int32_t *, int, int, int, double *,
                         const uint8_t *, int);
typedef void (*WideKernel)(const CUtensorMap *, int, float *, const int4 *, int, const int4 *, const int64_t *,
                           const float *, const int32_t *, int, int, int, double *, int, unsigned long long,
                           int, unsigned long long *, int, uint32_t *);

TbKernel tb_kernel(int depth) {
    switch (depth) {
    case 2: return k_sor32_tb<2>;
    case 4: return k_sor32_tb<4>;
    case 6: return k_sor32_tb<6>;
    default: return k_sor32_tb<8>;
    }
}

template <int W>
WideKernel wide_kernel_of(int depth) {
    switch (depth) {
    case 2: return k_sor32_wide<2, W>;
    case 4: return k_sor32_wide<4, W>;
    case 6: return k_sor32_wide<6, W>;
    default: return k_sor32_wide<8, W>;
    }
}

typedef void (*VolKernel)(const float *, float *, const float *, const float *, const int4 *, const int64_t *,
                          const int4 *, int, const float *, const int32_t *, int, int, int, double *, int);

template <int NW, int KIND>
VolKernel vol_kernel_of(int align) {
    return align == 16 ? k_sor32_vol<NW, 16, KIND> : align == 8 ? k_sor32_vol<NW, 8, KIND> : k_sor32_vol<NW, 4, KIND>;
}
template <int NW>
VolKernel vol_kernel_for(int align, int kind) {
    return kind == VOL_MIDDLE  ? vol_kernel_of<NW, VOL_MIDDLE>(align)
           : kind == VOL_FIRST ? vol_kernel_of<NW, VOL_FIRST>(align)
           : kind == VOL_LAST  ? vol_kernel_of<NW, VOL_LAST>(align)
                               : vol_kernel_of<NW, VOL_ANY>(align);
}
VolKernel vol_kernel(int vy, int align, int kind) {
    return vy == 16 ? vol_kernel_for<8>(align, kind) : vol_kernel_for<16>(align, kind);
}

WideKernel wide_kernel(int depth, int warps) {
    return warps * WROWS == 128 ? wide_kernel_of<128 / WROWS>(depth) : wide_kernel_of<64 / WROWS>(depth);
}

// Window starts along one axis of n pixels for windows of `win` with a halo
// of `depth`: the first at 0, then every win - 2 depth until one reaches n.
void axis_starts(int n, int win, int depth, std::vector<int> &out) {
    out.clear();
    out.push_back(0);
    if (n <= win) return;
    const int step = win - 2 * depth;
    const int last = (n - win + step - 1) / step;
    for (int k = 1; k <= last; ++k) out.push_back(k * step);
}

// The wide kernel's tensor maps, windows and grid, if every history allows it.
int wide_init(Sor32 &s, cw_field_s *f, int warps) {
    s.wide = false;
    s.wwarps = warps;
    const int WY = WROWS * warps;
    const size_t smem = wide_smem(warps);
    const Geom &g = f->g;
    for (uint32_t k = 0; k < g.nh; ++k)
        if (g.d[k] != 1 || g.w[k] % 4 != 0 || g.off[k] % 4 != 0) return CW_OK;
    if (s.depth % 2 != 0 || s.depth > 8) return CW_OK;
    PFN_cuTensorMapEncodeTiled_v12000 enc = tensor_map_encoder();
    if (!enc) return CW_OK;
    std::vector<CUtensorMap> maps(4 * (size_t)g.nh);
    float *arrays[4] = {f->d32a, f->d32b, f->r32, f->inv32};
    for (uint32_t k = 0; k < g.nh; ++k)
        for (int m = 0; m < 4; ++m) {
            cuuint64_t dim[2] = {(cuuint64_t)g.w[k], (cuuint64_t)g.h[k]};
            cuuint64_t stride[1] = {(cuuint64_t)g.w[k] * sizeof(float)};
            cuuint32_t box[2] = {(cuuint32_t)WX, (cuuint32_t)WY};
            cuuint32_t estride[2] = {1, 1};
            CUresult r = enc(&maps[4 * k + m], CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, arrays[m] + g.off[k], dim, stride,
                             box, estride, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                             CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
            if (r != CUDA_SUCCESS) return CW_OK;  // the narrow kernel serves
        }
    WideKernel kern = wide_kernel(s.depth, warps);
    if (cudaFuncSetAttribute((const void *)kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) !=
        cudaSuccess) {
        (void)cudaGetLastError();
        return CW_OK;  // the narrow kernel serves
    }
    int per_sm = 0, dev = 0, nsm = 0;
    CW_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, (const void *)kern, 32 * warps, smem));
    if (per_sm < 1) return CW_OK;
    CW_CUDA(cudaGetDevice(&dev));
    CW_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
    std::vector<int4> tiles;
    std::vector<int> xs, ys;
    for (uint32_t k = 0; k < g.nh; ++k) {
        axis_starts(g.w[k], WX, s.depth, xs);
        axis_starts(g.h[k], WY, s.depth, ys);
        for (int y : ys)
            for (int x : xs) tiles.push_back(make_int4((int)k, x, y, 0));
    }
    int rc;
    CUtensorMap *dm = nullptr;
    if ((rc = dalloc(&dm, maps.size())) != CW_OK) return rc;
    s.maps = dm;
    if ((rc = dalloc(&s.wtiles, tiles.size())) != CW_OK) return rc;
    CW_CUDA(cudaMemcpyAsync(s.maps, maps.data(), maps.size() * sizeof(CUtensorMap), cudaMemcpyHostToDevice,
                            stream()));
    CW_CUDA(cudaMemcpyAsync(s.wtiles, tiles.data(), tiles.size() * sizeof(int4), cudaMemcpyHostToDevice, stream()));
    CW_CUDA(cudaStreamSynchronize(stream()));
    s.nwtiles = (int)tiles.size();
    s.wgrid = std::min<int>(s.nwtiles, per_sm * nsm);
    s.wide = true;
    return CW_OK;
}

// The volume kernel's tiles: VX x vy columns (halo VD) by chunks of vz slices,
// an even number: the count of chunks whose waves of tiles march the fewest
// slices, halo and pipeline included (256^3: 275 tiles of 52 slices, two waves of
// 148, 66 steps each).
int vol_init(Sor32 &s, cw_field_s *f, int window) {
    s.vol = false;
    const Geom &g = f->g;
    int most = 0;
    s.valign = 16;
    for (uint32_t k = 0; k < g.nh; ++k) {
        if (g.d[k] < 2) return CW_OK;
        most = std::max(most, (int)g.d[k]);
        for (int64_t n : {(int64_t)g.w[k], g.off[k]})
            while (n * 4 % s.valign) s.valign /= 2;
    }
    s.vdepth = s.depth >= VD ? VD : 2;
    s.vy = window == CW_WINDOW_64 ? 16 : 32;
    const size_t smem = vol_smem(s.vy / 2);
    for (int kind : {VOL_ANY, VOL_MIDDLE, VOL_FIRST, VOL_LAST})
        CW_CUDA(cudaFuncSetAttribute((const void *)vol_kernel(s.vy, s.valign, kind),
                                     cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    int per_sm = 0, dev = 0, nsm = 0;
    CW_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, (const void *)vol_kernel(s.vy, s.valign, VOL_MIDDLE),
                                                          16 * s.vy, smem));
    if (per_sm < 1) return CW_OK;  // one half-sweep per launch serves
    CW_CUDA(cudaGetDevice(&dev));
    CW_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
    std::vector<int> xs, ys;
    std::vector<int64_t> columns(g.nh);
    for (uint32_t k = 0; k < g.nh; ++k) {
        axis_starts(g.w[k], VX, VD, xs);
        axis_starts(g.h[k], s.vy, VD, ys);
        columns[k] = (int64_t)xs.size() * ys.size();
    }
    const int64_t resident = (int64_t)per_sm * nsm;
    int64_t best = -1;
    for (int chunks = 1; chunks <= (most + 7) / 8; ++chunks) {
        const int vz = ((most + chunks - 1) / chunks + 1) / 2 * 2;
        int64_t n = 0;
        for (uint32_t k = 0; k < g.nh; ++k) n += columns[k] * ((g.d[k] + vz - 1) / vz);
        const int64_t cost = (n + resident - 1) / resident * (std::min(vz + 2 * VD, most) + VD + 2);
        if (best < 0 || cost < best) {
            best = cost;
            s.vz = vz;
        }
    }
    std::vector<int4> tiles;
    for (uint32_t k = 0; k < g.nh; ++k) {
        axis_starts(g.w[k], VX, VD, xs);
        axis_starts(g.h[k], s.vy, VD, ys);
        for (int z = 0; z < g.d[k]; z += s.vz)
            for (int y : ys)
                for (int x : xs) tiles.push_back(make_int4((int)k, x, y, z));
    }
    int rc;
    if ((rc = dalloc(&s.vtiles, tiles.size())) != CW_OK) return rc;
    CW_CUDA(cudaMemcpyAsync(s.vtiles, tiles.data(), tiles.size() * sizeof(int4), cudaMemcpyHostToDevice, stream()));
    CW_CUDA(cudaStreamSynchronize(stream()));
    s.nvtiles = (int)tiles.size();
    s.vol = true;
    return CW_OK;
}

}  // namespace

int Sor32::init(cw_field_s *f, int d, const std::vector<double> &om, int window) {
    depth = d < 1 ? 1 : d;
    if (depth > 1) depth = depth >= 8 ? 8 : (depth >= 6 ? 6 : (depth >= 4 ? 4 : 2));
    blocked = depth > 1;
    for (uint32_t k = 0; k < f->g.nh; ++k) blocked = blocked && f->g.d[k] == 1;
    std::vector<float> omf(om.begin(), om.end());
    int rc = dalloc(&omega, omf.size());
    if (rc != CW_OK) return rc;
    CW_CUDA(cudaMemcpyAsync(omega, omf.data(), sizeof(float) * omf.size(), cudaMemcpyHostToDevice, stream()));
    std::vector<int64_t> per(f->g.nh);
    if (blocked) {
        wide = false;
        if ((window == CW_WINDOW_AUTO || window == CW_WINDOW_TALL) &&
            (rc = wide_init(*this, f, window == CW_WINDOW_TALL ? 128 / WROWS : 64 / WROWS)) != CW_OK)
            return rc;
        if (!wide) {
            const int in = WIN - 2 * depth;
            for (uint32_t k = 0; k < f->g.nh; ++k)
                per[k] = (int64_t)((f->g.w[k] + in - 1) / in) * ((f->g.h[k] + in - 1) / in);
            rc = tiles.build(per, 1);
        }
    } else {
        vol = false;
        if (depth > 1 && (rc = vol_init(*this, f, window)) != CW_OK) return rc;
        if (!vol) {
            for (uint32_t k = 0; k < f->g.nh; ++k) per[k] = (int64_t)((f->g.w[k] + 1) / 2) * f->g.h[k] * f->g.d[k];
            rc = sites.build(per, 256);
        }
    }
    ping = f->d32a;
    pong = f->d32b;
    out = ping;
    return rc;
}

int Sor32::sweeps(cw_field_s *f, int n, const int32_t *done, int done_stride, float *start, bool apply,
                  unsigned long long *corr, int corr_stride) {
    if (apply && !wide && !vol && !blocked) 
        return fail(CW_ERR_CONFIG, "one half-sweep per launch applies no correction");
    if (start) {  // begin from this (zeroed) buffer; the other is scratch
        ping = start;
        pong = start == f->d32a ? f->d32b : f->d32a;
    }
    if (vol) {
        // 2n half-sweeps, vdepth per launch (fewer in the last), ping-pong
        // between the buffers; the first launch starts from zero
        float *a = ping, *b = pong;
        int remaining = 2 * n, done_half = 0;
        while (remaining > 0) {
            const int dd = remaining < vdepth ? remaining : vdepth;
            // with `apply` the last launch adds its correction to the field
            const bool last = remaining == dd;
            const bool adds = apply && last;
            const int kind = dd != VD || (adds && done_half == 0) ? VOL_ANY
                             : adds                              ? VOL_LAST
                             : done_half == 0                    ? VOL_FIRST
                                                                 : VOL_MIDDLE;
            CW_CUDA(launch_after(done_half > 0, vol_kernel(vy, valign, kind), nvtiles, 16 * vy, vol_smem(vy / 2),
                                 stream(), a, b, f->r32, f->inv32, f->g.d_dims, f->g.d_off, vtiles, vz, omega, done,
                                 done_stride, dd, done_half == 0 ? 1 : 0, apply && last ? f->c : nullptr,
                                 f->floor ? 1 : 0));
            CW_LAUNCHED();
            remaining -= dd;
            done_half += dd;
            float *t = a; a = b; b = t;
        }
        out = apply ? nullptr : a;
        return CW_OK;
    }
    if (!blocked) {
        for (int s = 0; s < n; ++s)
            for (int colour = 0; colour < 2; ++colour) {
                k_sor32_half<<<sites.nblocks, 256, 0, stream()>>>(ping, f->r32, f->inv32, f->g.d_dims, f->g.d_off,
                                                                  sites.d_blk, f->g.nh, omega, done, done_stride,
                                                                  colour);
                CW_LAUNCHED();
            }
        out = ping;
        return CW_OK;
    }
    // 2n half-sweeps, `depth` per launch (fewer in the last), starting from
    // the zeroed buffer; the windows are those of `depth`, whose halo is deep
    // enough for a shorter last launch too
    float *a = ping, *b = pong;
    int remaining = 2 * n, done_half = 0;
    while (remaining > 0) {
        int dd = remaining < depth ? remaining : depth;
        if (wide) {
            // the first launch starts from zero without reading it; with
            // `apply` the last adds its correction to the field
            const bool last = remaining == dd;
            CW_CUDA(launch_after(done_half > 0, wide_kernel(depth, wwarps), wgrid, 32 * wwarps, wide_smem(wwarps),
                                 stream(), (const CUtensorMap *)maps, a == f->d32a ? 0 : 1, b, wtiles, nwtiles, f->g.d_dims,
                                 f->g.d_off, omega, done, done_stride, dd, done_half == 0 ? 1 : 0,
                                 apply && last ? f->c : nullptr, f->floor ? 1 : 0,
                                 test_faults().wait_ns ? test_faults().wait_ns : TMA_WAIT_NS, test_faults().skip_tma,
                                 apply && last ? corr : nullptr, corr_stride, f->waits));
        } else {
            CW_CUDA(launch_after(done_half > 0, tb_kernel(depth), tiles.nblocks, 32 * WARPS, 0, stream(), a, b,
                                 f->r32, f->inv32, f->g.d_dims, f->g.d_off, tiles.d_blk, f->g.nh, omega, done,
                                 done_stride, dd, done_half == 0 ? 1 : 0, apply && remaining == dd ? f->c : nullptr,
                                 f->held, f->floor ? 1 : 0));
        }
        CW_LAUNCHED();
        remaining -= dd;
        done_half += dd;
        float *t = a; a = b; b = t;
    }
    out = apply ? nullptr : a;
    return CW_OK;
}

void Sor32::release() {
    dfree(omega);
    tiles.release();
    sites.release();
    CUtensorMap *m = (CUtensorMap *)maps;
    dfree(m);
    maps = nullptr;
    dfree(wtiles);
    wide = false;
    dfree(vtiles);
    vol = false;
}

}  // namespace cw
