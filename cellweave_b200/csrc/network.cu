// Protein network: Network of crates/engine/src/network.rs on the device.
//
// Compilation (from_spec, network.rs:283-445) runs once on the host: names
// are resolved to indices, terms laid out per node in file order.  The RK4
// step (rk4, network.rs:777-799) runs a lane per cell, a cell's nodes dealt to
// the warps of its block (k_rk4).
// Built without fused multiply-add: the sums round as the reference's do.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <map>
#include <string>

#include "cw_internal.cuh"
#include "network_kernels.cuh"

using namespace cw;

namespace {

const char *INPUTS[6] = {"oxygen", "egf", "crowding", "stress", "waste", "necrotic_factor"};

constexpr int MAXS = 32;

// Shared bytes of a k_rk4 block.
size_t rk4_block(int S, int nterms) {
    return sizeof(double) * (4 * S + 6) * RC + nterms * (sizeof(int4) + sizeof(double4)) + sizeof(int32_t) * (S + 1);
}

// RK4 with a block per 32 cells (rk4, derivatives and term_rate,
// network.rs:686-799): a lane per cell, the nodes dealt to the block's G warps.
// Every lane of a warp is at the same node, so a warp never diverges by kind of
// term, and a cell's evaluations run G nodes at a time.  A node's terms are
// added in file order by one thread: the reference's operations in its order.
// A stage's values live in shared memory, [node][lane], in two buffers turn by
// turn, so a stage is one barrier; the six inputs stand clamped behind them.
// Not CLONES: every cell under N, its terms in shared memory; else cell c under
// nets[clone[c]] (nets null: under N), its terms read from global memory (a
// network's tables are a few KB: they stay in L1).
// state: node i of cell c at state[i * node_stride + c * cell_stride], input q
// at inputs[q * in_stride + c * in_cell]; alive (optional): cells whose entry is
// zero are left as they are.
//
// What bounds it: with few cells the chain of a node's terms, each with a
// division; with many the FP64 instructions themselves.  A thread per cell (and
// for few cells a lane per node, whose warps diverged by kind of term) took, 10
// steps of 8 nodes: 300 cells 111 -> 49 us, 1,260 cells 115 -> 51, 16,000 cells
// 163 -> 72; 8 steps: 137,000 cells 452 -> 346, 40,000 cells of 16 nodes 693 ->
// 380, of 32 nodes 5,959 -> 1,204.  Five blocks of 8 warps an SM (48 registers a
// thread, a few of the power's spilled; four blocks spill next to none and take
// 445 us where five take 380).
template <int G, bool CLONES>
__global__ void __launch_bounds__(32 * G, 40 / G)
    k_rk4(NetDev N, const NetDev *nets, const int32_t *clone, int S, double *state, const double *inputs,
          int64_t ncells, int64_t node_stride, int64_t cell_stride, int64_t in_stride, int64_t in_cell, double dt,
          int substeps, const uint8_t *alive) {
    extern __shared__ double sm[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double *const xs = sm + lane, *const as = xs + S * RC, *const m0 = as + S * RC, *const m1 = m0 + S * RC,
                  *const in = m1 + S * RC;
    int4 *sterm = (int4 *)(sm + (4 * S + 6) * RC);
    double4 *spar = (double4 *)(sterm + N.nterms);
    int32_t *sptr = (int32_t *)(spar + N.nterms);
    const int64_t c = (int64_t)blockIdx.x * RC + lane;
    const bool live = c < ncells && !(alive && !alive[c]);
    const int4 *term = sterm;
    const double4 *par = spar;
    const int32_t *ptr = sptr;
    if (CLONES) {
        if (live) {
            const NetDev M = nets ? nets[clone[c]] : N;
            term = M.term;
            par = M.par;
            ptr = M.node_ptr;
        }
    } else {
        stage_terms(N, sterm, spar, sptr);
    }
    if (live) {
        for (int i = warp; i < S; i += G) xs[i * RC] = state[i * node_stride + c * cell_stride];
        for (int q = warp; q < 6; q += G) in[q * RC] = clamped_input(q, inputs[q * in_stride + c * in_cell]);
    }
    __syncthreads();
    auto rate_of = [&](const double *v, int i) { return node_rate<CLONES>(term, par, ptr, v, in, i); };
    for (int sub = 0; sub < substeps; ++sub) {
        // k1 at x, k2 at x + dt/2 k1, k3 at x + dt/2 k2, k4 at x + dt k3
        if (live)
            for (int i = warp; i < S; i += G) {
                const double k1 = rate_of(xs, i);
                as[i * RC] = k1;
                m0[i * RC] = xs[i * RC] + 0.5 * dt * k1;
            }
        __syncthreads();
        if (live)
            for (int i = warp; i < S; i += G) {
                const double k2 = rate_of(m0, i);
                as[i * RC] = as[i * RC] + 2.0 * k2;
                m1[i * RC] = xs[i * RC] + 0.5 * dt * k2;
            }
        __syncthreads();
        if (live)
            for (int i = warp; i < S; i += G) {
                const double k3 = rate_of(m1, i);
                as[i * RC] = as[i * RC] + 2.0 * k3;
                m0[i * RC] = xs[i * RC] + dt * k3;
            }
        __syncthreads();
        if (live)
            for (int i = warp; i < S; i += G) {
                const double acc = as[i * RC] + rate_of(m0, i);
                const double delta = (dt / 6.0) * acc;
                xs[i * RC] = fmin(fmax(xs[i * RC] + delta, 0.0), 1.0);
            }
        __syncthreads();
    }
    if (live)
        for (int i = warp; i < S; i += G) state[i * node_stride + c * cell_stride] = xs[i * RC];
}

template <int G, bool CLONES>
int rk4_launch(const NetDev &N, const NetDev *nets, const int32_t *clone, int S, double *state, const double *inputs,
               int64_t ncells, int64_t node_stride, int64_t cell_stride, int64_t in_stride, int64_t in_cell, double dt,
               int substeps, const uint8_t *alive) {
    k_rk4<G, CLONES><<<(unsigned)((ncells + RC - 1) / RC), 32 * G, rk4_block(S, CLONES ? 0 : N.nterms), stream()>>>(
        N, nets, clone, S, state, inputs, ncells, node_stride, cell_stride, in_stride, in_cell, dt, substeps, alive);
    CW_LAUNCHED();
    return CW_OK;
}

int rk4_cells(const NetDev &N, const NetDev *nets, const int32_t *clone, int S, double *state, const double *inputs,
              int64_t ncells, int64_t node_stride, int64_t cell_stride, int64_t in_stride, int64_t in_cell, double dt,
              int substeps, const uint8_t *alive) {
    int dev = 0, nsm = 0, most = 0;
    CW_CUDA(cudaGetDevice(&dev));
    CW_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
    CW_CUDA(cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
    // a network whose terms leave no room for a cell's columns beside them (one
    // node of 4,790 terms or more) reads them where they are
    const bool far = nets || rk4_block(S, N.nterms) > (size_t)most;
    const int64_t nblocks = (ncells + RC - 1) / RC;
    // A warp per node up to 16 while the blocks are few, for the shortest chain
    // (5,000 cells of 12 nodes 78 us against 120 with 8 warps); 8 warps where the
    // blocks fill the device, which then holds more cells at a time (40,000 cells
    // of 16 nodes 366 us against 425 with 16); 4 for many cells of few nodes, for
    // fewer warps at a barrier (400,000 cells of 8 nodes 918 us against 971 with 8).
    auto go = S > 8 && nblocks <= 2 * nsm     ? (far ? rk4_launch<16, true> : rk4_launch<16, false>)
              : S <= 8 && nblocks > 16 * nsm ? (far ? rk4_launch<4, true> : rk4_launch<4, false>)
                                             : (far ? rk4_launch<8, true> : rk4_launch<8, false>);
    return go(N, nets, clone, S, state, inputs, ncells, node_stride, cell_stride, in_stride, in_cell, dt, substeps,
              alive);
}

__global__ void k_mechanics(const double *state, int64_t ncells, int64_t stride, int growth, double coefficient,
                            double max_target, int has_max, uint32_t reference_volume, uint32_t *target) {
    int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= ncells) return;
    double g = state[growth * stride + c];
    double ratio = 1.0 + coefficient * g;
    if (has_max) ratio = fmin(ratio, max_target);
    double t = fmax((double)reference_volume * ratio, 0.0);
    target[c] = isnan(t) ? 0u : (t >= 4294967295.0 ? 4294967295u : (uint32_t)t);
}

// The most terms a network may have: what a block's shared memory would hold
// beside 64 cells' columns.
size_t network_bytes(const cw_network_s *n) {
    return sizeof(double) * 4 * n->S * 64 + n->nterms * (sizeof(int4) + sizeof(double4)) + sizeof(int32_t) * (n->S + 1);
}

// The device copies of a network's host tables (h_ptr, h_term, h_par).
int network_upload(cw_network_s *n) {
    n->nterms = (int32_t)n->h_term.size();
    int rc;
    if ((rc = dalloc(&n->node_ptr, n->S + 1)) || (rc = dalloc(&n->term, n->nterms)) ||
        (rc = dalloc(&n->par, n->nterms)))
        return rc;
    CW_CUDA(cudaMemcpy(n->node_ptr, n->h_ptr.data(), sizeof(int32_t) * (n->S + 1), cudaMemcpyHostToDevice));
    if (n->nterms > 0) {
        CW_CUDA(cudaMemcpy(n->term, n->h_term.data(), sizeof(int4) * n->nterms, cudaMemcpyHostToDevice));
        CW_CUDA(cudaMemcpy(n->par, n->h_par.data(), sizeof(double4) * n->nterms, cudaMemcpyHostToDevice));
    }
    int dev = 0, most = 0;
    CW_CUDA(cudaGetDevice(&dev));
    CW_CUDA(cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
    if (network_bytes(n) > (size_t)most)
        return fail(CW_ERR_CONFIG, "the network is too large for one block's shared memory");
    // (to the most there is, not to this network's need: it is the kernel's, whichever network it runs)
    if (rk4_block(n->S, n->nterms) > 48 * 1024) {
        for (auto k : {k_rk4<4, false>, k_rk4<8, false>, k_rk4<16, false>})
            CW_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
    }
    return CW_OK;
}

// A network like `n` with host tables to be changed and uploaded: every
// field but the device copies.
cw_network_s *network_derive(const cw_network_s *n) {
    cw_network_s *m = new cw_network_s();
    m->hs.init(false);
    m->S = n->S;
    m->names = n->names;
    m->initial = n->initial;
    std::memcpy(m->roles, n->roles, sizeof m->roles);
    m->growth_coefficient = n->growth_coefficient;
    m->lambda_volume = n->lambda_volume;
    m->max_target = n->max_target;
    m->reference_volume = n->reference_volume;
    m->h_ptr = n->h_ptr;
    m->h_term = n->h_term;
    m->h_par = n->h_par;
    return m;
}

// `(u * n as f64) as usize`, at most n - 1 (network.rs:488, 521): Rust's
// cast truncates and saturates (below zero and NaN give 0).
size_t pick_of(size_t n, double u) {
    if (n == 0) return 0;
    const double v = u * (double)n;
    if (!(v > 0.0)) return 0;
    if (v >= (double)n) return n - 1;
    return std::min<size_t>((size_t)v, n - 1);
}

// The node holding the term at global index t (terms in node order).
int node_of_term(const cw_network_s *n, int32_t t) {
    int i = 0;
    while (i + 1 < n->S && n->h_ptr[i + 1] <= t) ++i;
    return i;
}

constexpr double MUTATION_SPREAD = 2.0;  // network.rs:158
constexpr double GAINED_RATE = 0.1;      // network.rs:163
constexpr int REWIRED_INPUTS = 4;        // network.rs:169: oxygen, egf, crowding, stress

}  // namespace

namespace cw {
NetDev net_dev(const cw_network_s *n) { return NetDev{n->node_ptr, n->term, n->par, n->S, n->nterms}; }

// Device-side RK4 on node-major state (used by the simulation driver).
int network_step_device(const cw_network_s *n, double *state, const double *inputs, int64_t ncells,
                        int64_t state_stride, int64_t input_stride, double dt, int substeps, const uint8_t *alive) {
    if (ncells <= 0) return CW_OK;
    return rk4_cells(net_dev(n), nullptr, nullptr, n->S, state, inputs, ncells, state_stride, 1, input_stride, 1, dt,
                     substeps, alive);
}

// RK4 for cells of many networks on node-major state (the driver's evolving
// histories): cell c under nets[clone[c]], living cells only.
int network_step_clones_device(const NetDev *nets, const int32_t *clone, int S, double *state, const double *inputs,
                               int64_t ncells, int64_t state_stride, int64_t input_stride, double dt, int substeps,
                               const uint8_t *alive) {
    if (ncells <= 0) return CW_OK;
    NetDev none{};
    none.S = S;
    return rk4_cells(none, nets, clone, S, state, inputs, ncells, state_stride, 1, input_stride, 1, dt, substeps,
                     alive);
}

int network_mechanics_device(const cw_network_s *n, const double *state, int64_t ncells, int64_t stride,
                             uint32_t *target) {
    if (ncells <= 0) return CW_OK;
    bool has = !std::isnan(n->max_target);
    k_mechanics<<<(unsigned)((ncells + 255) / 256), 256, 0, stream()>>>(state, ncells, stride, n->roles[0],
                                                                       n->growth_coefficient,
                                                                       has ? n->max_target : 0.0, has ? 1 : 0,
                                                                       n->reference_volume, target);
    CW_LAUNCHED();
    return CW_OK;
}
int32_t network_nodes(const cw_network_s *n) { return n->S; }
double network_lambda(const cw_network_s *n) { return n->lambda_volume; }
int32_t network_role(const cw_network_s *n, int k) { return n->roles[k]; }
uint32_t network_reference_volume(const cw_network_s *n) { return n->reference_volume; }
const std::vector<double> &network_initial(const cw_network_s *n) { return n->initial; }
}  // namespace cw

extern "C" {

int cw_network_compile(int32_t nnodes, const char *const *names, const double *initial, int32_t nterms,
                       const cw_term_spec *terms, const char *growth, const char *survival, const char *hypoxia,
                       const char *differentiation, const char *apoptosis, const char *angiogenic,
                       const char *evasion, double growth_coefficient, double lambda_volume, double max_target,
                       uint32_t reference_volume, cw_network *out) {
    *out = nullptr;
    if (nnodes <= 0) return fail(CW_ERR_CONFIG, "a network needs a node");
    if (nnodes > MAXS) return fail(CW_ERR_CONFIG, "at most " + std::to_string(MAXS) + " nodes");
    if (!growth || !survival || !hypoxia)
        return fail(CW_ERR_CONFIG,
                    "the network declares no roles, and inherits none: say which node is growth, which is survival, "
                    "and which is the hypoxia response");
    std::map<std::string, int> index;
    for (int i = 0; i < nnodes; ++i) {
        std::string nm = names[i];
        for (auto in : INPUTS)
            if (nm == in)
                return fail(CW_ERR_CONFIG, "node `" + nm +
                                               "` takes the name of an environment input; inputs are [\"oxygen\", "
                                               "\"egf\", \"crowding\", \"stress\", \"waste\", \"necrotic_factor\"]");
        if (!index.emplace(nm, i).second) return fail(CW_ERR_CONFIG, "two nodes are named `" + nm + "`");
    }
    auto resolve = [&](const char *name, const std::string &whose, int32_t *src) -> int {
        std::string nm = name ? name : "";
        for (int q = 0; q < 6; ++q)
            if (nm == INPUTS[q]) { *src = -1 - q; return CW_OK; }
        auto it = index.find(nm);
        if (it != index.end()) { *src = it->second; return CW_OK; }
        std::string known = "[\"oxygen\", \"egf\", \"crowding\", \"stress\", \"waste\", \"necrotic_factor\"";
        for (int i = 0; i < nnodes; ++i) known += std::string(", \"") + names[i] + "\"";
        return fail(CW_ERR_CONFIG, "node `" + whose + "` reads `" + nm +
                                       "`, which is neither a node nor an input; known names are " + known + "]");
    };
    std::vector<int32_t> ptr(nnodes + 1, 0);
    std::vector<int4> tv(nterms);
    std::vector<double4> pv(nterms);
    int prev = 0;
    for (int t = 0; t < nterms; ++t) {
        const cw_term_spec &s = terms[t];
        if (s.node < prev || s.node >= nnodes) return fail(CW_ERR_CONFIG, "terms must be listed in node order");
        prev = s.node;
        ptr[s.node + 1] += 1;
        std::string whose = names[s.node];
        if (s.kind < CW_ACTIVATED_BY || s.kind > CW_DAMAGED_ABOVE)
            return fail(CW_ERR_CONFIG, "node `" + whose + "` has an unknown kind of term");
        int32_t src = 0;
        bool reads = s.kind != CW_DECAYS && s.kind != CW_RELAXES_TO;
        if (reads) {
            int rc = resolve(s.source, whose, &src);
            if (rc != CW_OK) return rc;
        }
        int has_hill = 0;
        if ((s.kind == CW_ACTIVATED_BY || s.kind == CW_INHIBITED_BY) && s.has_hill) {
            if (s.hill_n <= 0.0 || s.hill_k <= 0.0)
                return fail(CW_ERR_CONFIG, "node `" + whose + "` has a Hill term with n = " + std::to_string(s.hill_n) +
                                               " and k = " + std::to_string(s.hill_k) + "; both must be positive");
            has_hill = 1;
        }
        if ((s.kind == CW_DAMAGED_BELOW || s.kind == CW_DAMAGED_ABOVE) && s.param <= 0.0)
            return fail(CW_ERR_CONFIG, "node `" + whose + "` is damaged " +
                                           (s.kind == CW_DAMAGED_BELOW ? "below " : "above ") +
                                           std::to_string(s.param) + ", which must be positive");
        tv[t] = make_int4(s.kind, src, has_hill, 0);
        pv[t] = make_double4(s.rate, has_hill ? s.hill_n : 0.0, has_hill ? s.hill_k : 0.0, s.param);
    }
    for (int i = 0; i < nnodes; ++i) ptr[i + 1] += ptr[i];
    cw_network_s *n = new cw_network_s();
    if (n->hs.init(false) != CW_OK) { delete n; return CW_ERR_CUDA; }
    auto role = [&](const char *name, const char *which, int32_t *dst) -> int {
        if (!name) { *dst = -1; return CW_OK; }
        auto it = index.find(name);
        if (it == index.end())
            return fail(CW_ERR_CONFIG, std::string("the ") + which + " role names `" + name + "`, which is not a node");
        *dst = it->second;
        return CW_OK;
    };
    const char *rn[7] = {growth, survival, hypoxia, differentiation, apoptosis, angiogenic, evasion};
    const char *rw[7] = {"growth", "survival", "hypoxia response", "differentiation", "apoptosis", "angiogenic",
                         "evasion"};
    for (int k = 0; k < 7; ++k) {
        int rc = role(rn[k], rw[k], &n->roles[k]);
        if (rc != CW_OK) { delete n; return rc; }
    }
    n->S = nnodes;
    n->nterms = nterms;
    for (int i = 0; i < nnodes; ++i) {
        n->names.push_back(names[i]);
        double v = initial ? initial[i] : 0.0;
        n->initial.push_back(std::fmin(std::fmax(v, 0.0), 1.0));
    }
    n->growth_coefficient = growth_coefficient;
    n->lambda_volume = lambda_volume;
    n->max_target = max_target;
    n->reference_volume = reference_volume;
    n->h_ptr = ptr;
    n->h_term = tv;
    n->h_par = pv;
    int rc = network_upload(n);
    if (rc != CW_OK) {
        cw_network_destroy(n);
        return rc;
    }
    *out = n;
    return CW_OK;
}

int cw_network_destroy(cw_network n) {
    if (!n) return CW_OK;
    CW_SCOPE(n);
    dfree(n->node_ptr); dfree(n->term); dfree(n->par); dfree(n->cells.p);
    n->hs.release();
    delete n;
    return CW_OK;
}

int cw_network_set_stream(cw_network n, void *stream) {
    CW_SCOPE(n);
    return n->hs.set((cudaStream_t)stream);
}

void *cw_network_get_stream(cw_network n) { return (void *)n->hs.stream; }

const char *cw_network_last_error(cw_network n) { return n->hs.err.c_str(); }

int cw_network_info(cw_network n, int32_t *nnodes, int32_t *roles7, double *initial) {
    CW_SCOPE(n);
    if (nnodes) *nnodes = n->S;
    if (roles7) std::memcpy(roles7, n->roles, sizeof n->roles);
    if (initial) std::memcpy(initial, n->initial.data(), sizeof(double) * n->S);
    return CW_OK;
}

// The rows of a batch stay as the caller has them, [cell][node]: they are copied
// as they are and the kernel reads them at that stride (the transposes on the
// host and the allocations of each call took 3.3 of 4.0 ms for 40,000 cells of 16
// nodes, the kernel 0.7).
int cw_network_step_batch(cw_network n, int64_t ncells, double *state, const double *inputs, double dt,
                          int32_t substeps) {
    CW_SCOPE(n);
    if (ncells <= 0) return CW_OK;
    const int S = n->S;
    CellLease mem(n->cells);
    int rc;
    if ((rc = mem.take((size_t)ncells * (S + 6))) != CW_OK) return rc;
    double *d_state = mem.p, *d_in = d_state + ncells * S;
    CW_CUDA(cudaMemcpyAsync(d_state, state, sizeof(double) * ncells * S, cudaMemcpyHostToDevice, stream()));
    CW_CUDA(cudaMemcpyAsync(d_in, inputs, sizeof(double) * ncells * 6, cudaMemcpyHostToDevice, stream()));
    if ((rc = rk4_cells(net_dev(n), nullptr, nullptr, S, d_state, d_in, ncells, 1, S, 1, 6, dt, substeps, nullptr)) !=
        CW_OK)
        return rc;
    CW_CUDA(cudaMemcpyAsync(state, d_state, sizeof(double) * ncells * S, cudaMemcpyDeviceToHost, stream()));
    CW_CUDA(cudaStreamSynchronize(stream()));
    return CW_OK;
}

int cw_network_mechanics_batch(cw_network n, int64_t ncells, const double *state, uint32_t *target,
                               double *lambda) {
    CW_SCOPE(n);
    if (ncells <= 0) return CW_OK;
    const int S = n->S;
    double *d_state;
    uint32_t *d_t;
    int rc;
    if ((rc = dalloc(&d_state, (size_t)ncells * S)) || (rc = dalloc(&d_t, (size_t)ncells))) return rc;
    std::vector<double> t((size_t)ncells * S);
    for (int64_t c = 0; c < ncells; ++c)
        for (int i = 0; i < S; ++i) t[(size_t)i * ncells + c] = state[c * S + i];
    CW_CUDA(cudaMemcpyAsync(d_state, t.data(), sizeof(double) * ncells * S, cudaMemcpyHostToDevice, stream()));
    if ((rc = network_mechanics_device(n, d_state, ncells, ncells, d_t)) != CW_OK) return rc;
    CW_CUDA(cudaMemcpyAsync(target, d_t, sizeof(uint32_t) * ncells, cudaMemcpyDeviceToHost, stream()));
    CW_CUDA(cudaStreamSynchronize(stream()));
    if (lambda)
        for (int64_t c = 0; c < ncells; ++c) lambda[c] = n->lambda_volume;
    dfree(d_state);
    dfree(d_t);
    return CW_OK;
}

int cw_network_mutate(cw_network n, double which, double how, cw_network *out, cw_mutation *rec) {
    CW_SCOPE(n);
    if (!out) return fail(CW_ERR_CONFIG, "no place for the mutated network");
    *out = nullptr;
    const size_t count = n->h_term.size();
    if (count == 0) return fail(CW_ERR_NOT_FOUND, "a network without a single term has nothing a mutation could change");
    const int32_t pick = (int32_t)pick_of(count, which);
    const double factor = std::pow(MUTATION_SPREAD, 2.0 * how - 1.0);
    cw_network_s *m = network_derive(n);
    m->h_par[pick].x = m->h_par[pick].x * factor;
    const int node = node_of_term(n, pick);
    int rc = network_upload(m);
    if (rc != CW_OK) {
        cw_network_destroy(m);
        return rc;
    }
    if (rec) *rec = cw_mutation{node, pick - n->h_ptr[node], n->h_term[pick].x, CW_CHANGE_SCALED, factor, 0, 0};
    *out = m;
    return CW_OK;
}

int cw_network_rewire(cw_network n, const double draws[5], cw_network *out, cw_mutation *rec) {
    CW_SCOPE(n);
    if (!out || !draws) return fail(CW_ERR_CONFIG, "rewiring takes five draws and a place for the network");
    *out = nullptr;
    const double mode = draws[0], which = draws[1], source = draws[2], sign = draws[3], how = draws[4];
    cw_network_s *m = network_derive(n);
    cw_mutation r{};
    if (mode < 0.5) {
        // a gained link, the node's last term
        const int node = (int)pick_of((size_t)n->S, which);
        const int s = (int)pick_of((size_t)(REWIRED_INPUTS + n->S), source);
        const int32_t src = s < REWIRED_INPUTS ? -1 - s : s - REWIRED_INPUTS;
        const double rate = GAINED_RATE * std::pow(MUTATION_SPREAD, 2.0 * how - 1.0);
        const int32_t kind = sign < 0.5 ? CW_ACTIVATED_BY : CW_ACTIVATED_BY_ABSENCE_OF;
        const int32_t at = m->h_ptr[node + 1];
        m->h_term.insert(m->h_term.begin() + at, make_int4(kind, src, 0, 0));
        m->h_par.insert(m->h_par.begin() + at, make_double4(rate, 0.0, 0.0, 0.0));
        for (int i = node + 1; i <= n->S; ++i) m->h_ptr[i] += 1;
        r = cw_mutation{node, at - n->h_ptr[node], kind, CW_CHANGE_GAINED, rate, src, 0};
    } else {
        const size_t count = n->h_term.size();
        if (count == 0) {
            delete m;
            return fail(CW_ERR_NOT_FOUND, "a network without a single term has no term to lose");
        }
        const int32_t at = (int32_t)pick_of(count, which);
        const int node = node_of_term(n, at);
        r = cw_mutation{node, at - n->h_ptr[node], n->h_term[at].x, CW_CHANGE_LOST, 0.0, 0, 0};
        m->h_term.erase(m->h_term.begin() + at);
        m->h_par.erase(m->h_par.begin() + at);
        for (int i = node + 1; i <= n->S; ++i) m->h_ptr[i] -= 1;
    }
    int rc = network_upload(m);
    if (rc != CW_OK) {
        cw_network_destroy(m);
        return rc;
    }
    if (rec) *rec = r;
    *out = m;
    return CW_OK;
}

int cw_network_step_clones(int32_t nnets, const cw_network *nets, int64_t ncells, const int32_t *clone,
                           double *state, const double *inputs, double dt, int32_t substeps) {
    if (ncells <= 0) return CW_OK;
    if (nnets <= 0 || !nets) return fail(CW_ERR_CONFIG, "no networks to step the cells under");
    const int S = nets[0]->S;
    std::vector<NetDev> dev(nnets);
    for (int k = 0; k < nnets; ++k) {
        if (!nets[k] || nets[k]->S != S) return fail(CW_ERR_CONFIG, "every network of a batch has the same nodes");
        dev[k] = net_dev(nets[k]);
    }
    for (int64_t c = 0; c < ncells; ++c)
        if (clone[c] < 0 || clone[c] >= nnets)
            return fail(CW_ERR_CONFIG, "cell " + std::to_string(c) + " names network " + std::to_string(clone[c]) +
                                           " of " + std::to_string(nnets));
    CellLease mem(nets[0]->cells);
    const size_t nets_at = (size_t)ncells * (S + 6), clone_at = nets_at + (sizeof(NetDev) * nnets + 7) / 8;
    int rc;
    if ((rc = mem.take(clone_at + (size_t)(ncells + 1) / 2)) != CW_OK) return rc;
    double *d_state = mem.p, *d_in = d_state + ncells * S;
    NetDev *d_nets = (NetDev *)(mem.p + nets_at);
    int32_t *d_clone = (int32_t *)(mem.p + clone_at);
    CW_CUDA(cudaMemcpyAsync(d_state, state, sizeof(double) * ncells * S, cudaMemcpyHostToDevice, stream()));
    CW_CUDA(cudaMemcpyAsync(d_in, inputs, sizeof(double) * ncells * 6, cudaMemcpyHostToDevice, stream()));
    CW_CUDA(cudaMemcpyAsync(d_nets, dev.data(), sizeof(NetDev) * nnets, cudaMemcpyHostToDevice, stream()));
    CW_CUDA(cudaMemcpyAsync(d_clone, clone, sizeof(int32_t) * ncells, cudaMemcpyHostToDevice, stream()));
    NetDev none{};
    none.S = S;
    if ((rc = rk4_cells(none, d_nets, d_clone, S, d_state, d_in, ncells, 1, S, 1, 6, dt, substeps, nullptr)) != CW_OK)
        return rc;
    CW_CUDA(cudaMemcpyAsync(state, d_state, sizeof(double) * ncells * S, cudaMemcpyDeviceToHost, stream()));
    CW_CUDA(cudaStreamSynchronize(stream()));
    return CW_OK;
}

}  // extern "C"
