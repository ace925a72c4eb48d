// The compiled network and its device-side term evaluation, shared by the
// RK4 step (network.cu) and its adjoint (adjoint.cu).
#pragma once

#include <cmath>
#include <mutex>
#include <string>
#include <vector>

#include "cw_internal.cuh"

namespace cw {

// A network's device memory for the batches of cells that come from the host:
// kept up to KEPT bytes, given back with the network.  One call at a time has it;
// a call that finds it taken (another thread's on the same network), or that needs
// more, allocates its own for its own time.
struct CellSpace {
    static constexpr size_t KEPT = (size_t)64 << 20;
    std::mutex mu;
    double *p = nullptr;
    size_t bytes = 0;
};
class CellLease {
  public:
    explicit CellLease(CellSpace &s) : s_(s), lock_(s.mu, std::try_to_lock) {}
    CellLease(const CellLease &) = delete;
    CellLease &operator=(const CellLease &) = delete;
    // what the call queued is over before the memory is another's
    ~CellLease() {
        if (p) cudaStreamSynchronize(stream());
        dfree(own_);
    }
    int take(size_t numbers) {
        const size_t bytes = numbers * sizeof(double);
        int rc = CW_OK;
        if (!lock_.owns_lock() || bytes > CellSpace::KEPT) {
            if ((rc = dalloc(&own_, numbers)) == CW_OK) p = own_;
            return rc;
        }
        if (bytes > s_.bytes) {
            dfree(s_.p);
            s_.bytes = 0;
            if ((rc = dalloc(&s_.p, numbers)) != CW_OK) return rc;
            s_.bytes = bytes;
        }
        p = s_.p;
        return CW_OK;
    }
    double *p = nullptr;

  private:
    CellSpace &s_;
    std::unique_lock<std::mutex> lock_;
    double *own_ = nullptr;
};

}  // namespace cw

struct cw_network_s {
    cw::HandleStream hs;  // its stream and last error
    int32_t S = 0, nterms = 0;
    std::vector<std::string> names;
    std::vector<double> initial;
    int32_t roles[7] = {-1, -1, -1, -1, -1, -1, -1};
    double growth_coefficient = 0.0, lambda_volume = 0.0, max_target = NAN;
    uint32_t reference_volume = 0;
    // the compiled terms on the host (node_ptr, term, par below), for the
    // mutations that derive a network from this one
    std::vector<int32_t> h_ptr;
    std::vector<int4> h_term;
    std::vector<double4> h_par;
    // device copies of the compiled terms
    int32_t *node_ptr = nullptr;  // S + 1
    int4 *term = nullptr;         // (kind, source, has_hill, 0)
    double4 *par = nullptr;       // (rate, hill_n, hill_k, param)
    cw::CellSpace cells;
};

namespace cw {

struct NetDev {
    const int32_t *node_ptr;
    const int4 *term;
    const double4 *par;
    int32_t S, nterms;
};

// read, network.rs:670-680.
__device__ __forceinline__ double read_source(int32_t src, const double *in, const double *st, int stride) {
    if (src >= 0) return st[src * stride];
    switch (-1 - src) {
    case 0: return fmin(fmax(in[0], 0.0), 1.0);
    case 1: return in[1];
    case 2: return fmin(fmax(in[2], 0.0), 1.0);
    case 3: return fmax(in[3], 0.0);
    case 4: return fmax(in[4], 0.0);
    default: return fmax(in[5], 0.0);
    }
}

// driver, network.rs:56-64.  A Hill exponent of exactly two is a square.
__device__ __forceinline__ double hill(double s, double n, double half) {
    double sp = fmax(s, 0.0);
    double sn, hn;
    if (n == 2.0) { sn = sp * sp; hn = half * half; }
    else { sn = pow(sp, n); hn = pow(half, n); }
    return sn / (hn + sn);
}

// derivatives + term_rate, network.rs:686-734, for the thread's cell.
// st/out point at node 0 of this thread's column (stride = threads).
__device__ __forceinline__ void derivatives(const NetDev &N, const int4 *sterm, const double4 *spar, const int32_t *sptr,
                            const double *st, const double *in, double *out, int stride) {
    for (int i = 0; i < N.S; ++i) {
        double own = st[i * stride], rate = 0.0;
        for (int t = sptr[i]; t < sptr[i + 1]; ++t) {
            int4 tm = sterm[t];
            double4 p = spar[t];
            double k = p.x, r;
            switch (tm.x) {
            case CW_ACTIVATED_BY: {
                double s = read_source(tm.y, in, st, stride);
                double drv = tm.z ? hill(s, p.y, p.z) : s;
                r = k * drv * (1.0 - own);
                break;
            }
            case CW_INHIBITED_BY: {
                double s = read_source(tm.y, in, st, stride);
                double drv = tm.z ? hill(s, p.y, p.z) : s;
                r = -k * drv * own;
                break;
            }
            case CW_ACTIVATED_BY_ABSENCE_OF:
                r = k * (1.0 - read_source(tm.y, in, st, stride)) * (1.0 - own);
                break;
            case CW_PRODUCED_BY: r = k * read_source(tm.y, in, st, stride); break;
            case CW_DECAYS: r = -k * own; break;
            case CW_RELAXES_TO: r = -k * (own - p.w); break;
            case CW_DAMAGED_BELOW: {
                double s = read_source(tm.y, in, st, stride);
                r = -k * fmax((p.w - s) / p.w, 0.0);
                break;
            }
            default: {
                double s = read_source(tm.y, in, st, stride);
                r = -k * fmax((s - p.w) / p.w, 0.0);
                break;
            }
            }
            rate += r;
        }
        out[i * stride] = rate;
    }
}

// ------------------------------------------------------------------ a lane per cell, a cell's nodes over warps
constexpr int RC = 32;           // cells per block: the stride of a column
enum { SQUARE = 2, POWER = 3 };  // a staged term's Hill flag

// read, network.rs:670-680: oxygen and crowding in [0, 1], stress and the
// released not below zero.
__device__ __forceinline__ double clamped_input(int q, double v) {
    return q == 0 || q == 2 ? fmin(fmax(v, 0.0), 1.0) : q >= 3 ? fmax(v, 0.0) : v;
}

// A network's terms into shared memory, what a Hill response takes from its
// term alone worked out: the flag says how s is raised, par.z is the half's power.
__device__ __forceinline__ void stage_terms(const NetDev &N, int4 *sterm, double4 *spar, int32_t *sptr) {
    for (int t = threadIdx.x; t < N.nterms; t += blockDim.x) {
        int4 tm = N.term[t];
        double4 p = N.par[t];
        if (tm.z) {
            tm.z = p.y == 2.0 ? SQUARE : POWER;
            p.z = p.y == 2.0 ? p.z * p.z : pow(p.z, p.y);
        }
        sterm[t] = tm;
        spar[t] = p;
    }
    for (int t = threadIdx.x; t <= N.S; t += blockDim.x) sptr[t] = N.node_ptr[t];
}

// A term's source from the lane's columns: node values v, clamped inputs in.
__device__ __forceinline__ double source_of(const int4 &tm, const double *v, const double *in) {
    return tm.y >= 0 ? v[tm.y * RC] : in[min(-1 - tm.y, 5) * RC];
}

// The rate of node i at the lane's values v (derivatives and term_rate,
// network.rs:686-734), its terms added in file order; RAW: tables as compiled,
// else as stage_terms leaves them.
template <bool RAW>
__device__ __forceinline__ double node_rate(const int4 *term, const double4 *par, const int32_t *ptr, const double *v,
                                            const double *in, int i) {
    const double own = v[i * RC], rest = 1.0 - own;
    double rate = 0.0;
    const int end = ptr[i + 1];
    for (int t = ptr[i]; t < end; ++t) {
        const int4 tm = term[t];
        const double4 p = par[t];
        const double s = source_of(tm, v, in);
        const double k = p.x;
        double r;
        switch (tm.x) {
        case CW_ACTIVATED_BY:
        case CW_INHIBITED_BY: {
            double drv = s;
            if (RAW) {
                if (tm.z) drv = hill(s, p.y, p.z);
            } else if (tm.z) {  // driver, network.rs:56-64
                const double sp = s > 0.0 ? s : 0.0;
                const double sn = tm.z == SQUARE ? sp * sp : pow(sp, p.y);
                drv = sn / (p.z + sn);
            }
            r = tm.x == CW_ACTIVATED_BY ? k * drv * rest : -k * drv * own;
            break;
        }
        case CW_ACTIVATED_BY_ABSENCE_OF: r = k * (1.0 - s) * rest; break;
        case CW_PRODUCED_BY: r = k * s; break;
        case CW_DECAYS: r = -k * own; break;
        case CW_RELAXES_TO: r = -k * (own - p.w); break;
        case CW_DAMAGED_BELOW: r = -k * fmax((p.w - s) / p.w, 0.0); break;
        default: r = -k * fmax((s - p.w) / p.w, 0.0); break;
        }
        rate += r;
    }
    return rate;
}

}  // namespace cw
