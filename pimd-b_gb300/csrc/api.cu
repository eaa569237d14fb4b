// C ABI (include/pimdb_gb300.h): handle lifetime, state transfer and the
// per-step schedule of kernels on one CUDA stream.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <map>
#include <new>
#include <tuple>
#include <string>
#include <vector>

#include "../../include/pimdb_gb300.h"
#include "common.cuh"
#include "config.h"
#include "kernels.h"

using namespace pimdb;

struct pimdb_handle {
    pimdb_config cfg;
    int D = 3;
    Sys s{};
    cudaStream_t stream = nullptr;
    bool own_stream = false;
    // second stream: the exchange chain (latency-bound, two blocks) runs
    // beside the pair forces (throughput-bound, every SM)
    cudaStream_t side = nullptr;
    cudaEvent_t fork_ev = nullptr, join_ev = nullptr;
    double* d_C = nullptr;    // cart -> NM rows [P][P]
    double* d_T = nullptr;    // NM -> cart rows [P][P]
    double* d_rot = nullptr;  // [P][4]: cos, sin, m omega_k, sin / (m omega_k)
    double* d_red[2] = {nullptr, nullptr};
    double* d_stage = nullptr;
    double* d_part = nullptr;  // pair-tile partial sums (Newton's third law path)
    double* d_obs = nullptr;   // the energy and observable terms (obs_work), from the first call on
    int* d_err = nullptr;
    long long step = 0;
    // coordinate generation: advanced by every call that can change x; the
    // split exchange's adjoint and dbeta need the forward of the current one
    long long xgen = 0, fwd_gen = -1;
    int red_last = 0;         // buffer holding the pending COM partials
    int nred_last = 0;
    bool com_pending = false;
    std::string last_error;
    // instrumentation: kernel launch count and, when enabled, per-class
    // device time measured with events bracketing each launch
    long long launches = 0;
    int opt_exact_exchange = 0;
    // fused normal-mode step (normal-mode propagator + normal-mode thermostat)
    bool fused_nm = false;
    bool nm_tail_pending = false;
    double* d_cmpart = nullptr;
    unsigned* d_bar = nullptr;
    double* d_tw = nullptr;   // FFT twiddles (P/2 complex) when P is a power of two
    // the normal modes of p and x the last fused head left (three-warp
    // kernel), valid while nothing else has changed x or p
    double* d_modes = nullptr;
    bool modes_valid = false;
    int logP = 0;
    int opt_fft = 1;
    cudaError_t async_err = cudaSuccess;
    int opt_newton3 = 1;
    int opt_reserved_sms = -1;  // SMs the pair tiles leave to the exchange (-1: by exchange size)
    // cell lists (periodic box with a short cutoff): cells per edge, work
    // buffer, and the option (-1 automatic: on when nc >= 4 and N >= 512)
    int cell_nc = 0;
    void* d_cells = nullptr;
    // Nose-Hoover chains: parameters and state (eta, eta_dot, eta_dot_dot),
    // and the normal-mode momenta buffer of the normal-mode coupling
    NHPar nh{};
    long long nh_chains = 0;
    double* d_nh = nullptr;
    double* d_pnm = nullptr;
    int opt_cells = -1;
    bool factorial = false;  // the exchange is the sum over all N! permutations
    // RanMars parity noise: the streams and the staged normals (Sys::noise)
    RanMarsState* d_rng = nullptr;
    double* d_noise = nullptr;
    int* h_err = nullptr;  // pinned copy of the error word
    // the exchange's triangular solve across SMs (large N): y of both
    // directions and the publication flags
    double* d_ysol = nullptr;
    double* d_ework = nullptr;  // link prefix sums and wrapped end beads (large N)
    unsigned* d_gflags = nullptr;
    // CUDA graphs of pimdb_step_async: keyed by the step count and the
    // host-side step state at entry; the step index comes from d_step, which
    // every graph advances by its step count
    struct StepState {
        int red_last, nred_last;
        bool com_pending, nm_tail_pending, modes_valid;
        bool operator<(const StepState& o) const {
            return std::tie(red_last, nred_last, com_pending, nm_tail_pending, modes_valid) <
                   std::tie(o.red_last, o.nred_last, o.com_pending, o.nm_tail_pending, o.modes_valid);
        }
    };
    struct StepGraph {
        cudaGraphExec_t exec = nullptr;
        StepState after{};
        long long kernels = 0;
    };
    std::map<std::pair<int, StepState>, StepGraph> graphs;
    // whole pimdb_step_io calls on page-locked buffers: (steps, state before,
    // device views of x_in, p_in, x_out, p_out, f_out)
    struct IoKey {
        int nsteps;
        StepState before;
        const void* v[5];
        bool operator<(const IoKey& o) const {
            return std::tie(nsteps, before, v[0], v[1], v[2], v[3], v[4]) <
                   std::tie(o.nsteps, o.before, o.v[0], o.v[1], o.v[2], o.v[3], o.v[4]);
        }
    };
    std::map<IoKey, StepGraph> io_graphs;
    long long* d_step = nullptr;
    bool dstep_valid = false;
    bool capturing = false;
    long long graph_base = 0;
    int opt_graph = 1;
    bool graph_broken = false;
    bool warm = false;  // one uncaptured step first: lazy attribute and occupancy set-up stays out of captures
    bool profile = false;
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
    double prof_ms[PIMDB_NUM_KERNEL_CLASSES] = {};
    long long prof_n[PIMDB_NUM_KERNEL_CLASSES] = {};
};

// Enqueues one kernel launch of class `cls` on the handle's stream.
template <class F>
static void launch(pimdb_handle* h, int cls, F&& f, int nkernels = 1) {
    h->launches += nkernels;
    if (!h->profile) {
        f();
        return;
    }
    cudaEventRecord(h->ev0, h->stream);
    f();
    cudaEventRecord(h->ev1, h->stream);
    cudaEventSynchronize(h->ev1);
    float ms = 0.f;
    cudaEventElapsedTime(&ms, h->ev0, h->ev1);
    h->prof_ms[cls] += ms;
    h->prof_n[cls] += 1;
}

// Step index argument of a launch: absolute, or relative to the graph's
// start while a graph is being captured.
static StepRef step_ref(const pimdb_handle* h, long long step) {
    if (h->capturing) return StepRef{h->d_step, step - h->graph_base};
    return StepRef{nullptr, step};
}

// The last node of a step graph: the device step counter moves on.
__global__ void k_step_advance(long long* step, int n) { *step += n; }
static void launch_step_advance(long long* step, int n, cudaStream_t st) { k_step_advance<<<1, 1, 0, st>>>(step, n); }

static void drop_graphs(pimdb_handle* h) {
    for (auto& kv : h->graphs)
        if (kv.second.exec) cudaGraphExecDestroy(kv.second.exec);
    h->graphs.clear();
    for (auto& kv : h->io_graphs)
        if (kv.second.exec) cudaGraphExecDestroy(kv.second.exec);
    h->io_graphs.clear();
}

static void complete_pending(pimdb_handle* h);

static std::string g_last_error;

static int fail(pimdb_handle* h, int code, const std::string& msg) {
    if (h) h->last_error = msg;
    g_last_error = msg;
    return code;
}

#define CUDA_TRY(h, expr)                                                                       \
    do {                                                                                        \
        cudaError_t e_ = (expr);                                                                \
        if (e_ != cudaSuccess) return fail((h), PIMDB_ERR_CUDA, std::string(#expr ": ") + cudaGetErrorString(e_)); \
    } while (0)

extern "C" const char* pimdb_status_string(int st) {
    switch (st) {
    case PIMDB_OK: return "ok";
    case PIMDB_ERR_CONFIG: return "invalid configuration";
    case PIMDB_ERR_NONFINITE_VB: return "non-finite bosonic exchange potential";
    case PIMDB_ERR_CUDA: return "CUDA error";
    case PIMDB_ERR_TIMEOUT: return "device wait timed out";
    case PIMDB_ERR_BOUNDS: return "device index out of bounds";
    case PIMDB_ERR_ARG: return "invalid argument";
    case PIMDB_ERR_NO_DEVICE: return "no CUDA device";
    case PIMDB_ERR_PARSE: return "cannot read configuration file";
    default: return "unknown status";
    }
}

extern "C" int pimdb_last_error(const pimdb_handle* h, char* buf, int len) {
    if (!buf || len <= 0) return PIMDB_ERR_ARG;
    const std::string& m = h ? h->last_error : g_last_error;
    std::snprintf(buf, (size_t)len, "%s", m.c_str());
    return PIMDB_OK;
}

extern "C" int pimdb_config_default(pimdb_config* c) {
    if (!c) return PIMDB_ERR_ARG;
    std::memset(c, 0, sizeof(*c));
    // src/params.cpp:15-259 defaults
    c->ndim = 3;
    c->natoms = 1;
    c->nbeads = 4;
    c->fixcom = 1;
    c->dt = 1.0 * 4.1341373e16 * 1e-15;        // 1 femtosecond
    c->gamma = -1.0;
    c->temperature = 1.0 * 3.1668152e-06;      // 1 kelvin
    c->mass = 1.0 * 1822.8885;                 // 1 dalton
    c->size = 1.0 * 1.8897261e10 * 1e-12;      // 1 picometer
    c->cutoff = -1.0 * 1.8897261;              // -1 angstrom
    c->seed = 1234;
    c->thermostat = PIMDB_THERMO_LANGEVIN;
    c->nchains = 4;
    return PIMDB_OK;
}

std::string validate_config(const pimdb_config& c) {
    if (c.ndim < 1 || c.ndim > 3) return "ndim must be 1, 2 or 3";
    if (c.nbeads < 1) return "The specified number of beads is less than one!";
    if (c.natoms < 1) return "The specified number of particles is smaller than one!";
    if (!(c.temperature > 0.0)) return "The specified temperature is unphysical!";
    if (!(c.mass > 0.0)) return "The provided mass is unphysical!";
    if (!(c.size > 0.0)) return "The provided system size is unphysical!";
    if (!(c.dt > 0.0)) return "dt must be positive";
    if (c.propagator != PIMDB_PROP_CARTESIAN && c.propagator != PIMDB_PROP_NORMAL_MODES)
        return "The specified time propagator is not supported!";
    if (c.thermostat < PIMDB_THERMO_NONE || c.thermostat > PIMDB_THERMO_NOSE_HOOVER_NP_DIM)
        return "The specified thermostat is not supported!";
    if (c.thermostat >= PIMDB_THERMO_NOSE_HOOVER && c.nchains < 1)
        return "The specified number of Nose-Hoover chains (" + std::to_string(c.nchains) + ") is less than one!";
    if (c.nmthermostat && c.thermostat == PIMDB_THERMO_NONE) return "nmthermostat cannot be used in nve ensemble!";
    if (c.ext_kind != PIMDB_POT_FREE && c.ext_kind != PIMDB_POT_HARMONIC && c.ext_kind != PIMDB_POT_DOUBLE_WELL &&
        c.ext_kind != PIMDB_POT_COSINE)
        return "The specified external potential is not supported!";
    if (c.int_kind != PIMDB_POT_FREE && c.int_kind != PIMDB_POT_HARMONIC && c.int_kind != PIMDB_POT_AZIZ &&
        c.int_kind != PIMDB_POT_DIPOLE)
        return "The specified interaction potential is not supported!";
    if (c.precision != PIMDB_FP64 && c.precision != PIMDB_MIXED) return "unknown precision";
    if ((long long)c.natoms * c.nbeads * c.ndim > (1ll << 31)) return "system too large";
    if ((c.propagator == PIMDB_PROP_NORMAL_MODES || c.nmthermostat) && c.nbeads > kNmMaxBeads)
        return "normal modes support at most " + std::to_string(kNmMaxBeads) + " beads";
    if (c.bosonic && c.nbeads > 1 && c.natoms > kExchangeMaxN)
        return "bosonic exchange supports at most " + std::to_string(kExchangeMaxN) + " particles";
    if (c.exchange != PIMDB_EXCHANGE_FELDMAN_HIRSHBERG && c.exchange != PIMDB_EXCHANGE_FACTORIAL)
        return "unknown bosonic exchange algorithm";
    if (c.exchange == PIMDB_EXCHANGE_FACTORIAL && c.bosonic && c.nbeads > 1 && c.natoms > kFactMaxN)
        return "the factorial bosonic exchange supports at most " + std::to_string(kFactMaxN) + " particles";
    if (c.rng != PIMDB_RNG_PHILOX && c.rng != PIMDB_RNG_RANMAR) return "unknown noise generator";
    // RanMars(params_seed + rank) for every bead (simulation.cpp:59, random_mars.cpp:16-17)
    if (c.rng == PIMDB_RNG_RANMAR && (c.seed < 1 || c.seed + (unsigned long long)c.nbeads - 1 > 900000000ull))
        return "Invalid seed for Marsaglia random # generator";
    return "";
}

void sys_params_from_config(const pimdb_config& c, Sys& s) {
    s.N = c.natoms;
    s.eflat = exchange_flat_default(c.natoms);
    s.P = c.nbeads;
    s.ld = (c.natoms + 31) / 32 * 32;
    s.bosonic = (c.bosonic && c.nbeads > 1) ? 1 : 0;  // simulation.cpp:690
    s.pbc = c.pbc ? 1 : 0;
    s.L = c.size;
    s.invL = 1.0 / c.size;
    s.mass = c.mass;
    s.dt = c.dt;
    s.dt_m = c.dt / c.mass;
    // simulation.cpp:37-52 (IPI convention, kB = hbar = 1)
    const double beta = 1.0 / (1.0 * c.temperature);
    const double thermo_beta = beta / c.nbeads;
    s.omega_p = c.nbeads / (beta * 1.0);
    s.kappa = c.mass * s.omega_p * s.omega_p;
    s.beta_ex = beta / c.nbeads;  // bosonic_exchange_base.cpp:16-18
    s.inv_beta_ex = 1.0 / s.beta_ex;
    // langevin.cpp:11-12, params.cpp:17-20
    const double gamma = c.gamma < 0 ? 1 / (100.0 * c.dt) : c.gamma;
    s.c1 = std::exp(-0.5 * gamma * c.dt);
    s.c2 = std::sqrt((1 - s.c1 * s.c1) * c.mass / thermo_beta);
    // simulation.cpp:84-90
    double cut = (c.int_kind == PIMDB_POT_FREE) ? 0.0 : c.cutoff;
    if (c.pbc && 0.5 * c.size < cut) cut = 0.5 * c.size;
    s.cutoff = cut;
    s.ext_kind = c.ext_kind;
    if (c.ext_kind == PIMDB_POT_HARMONIC) {
        s.ext_a = c.mass * c.ext_params[0] * c.ext_params[0];
    } else if (c.ext_kind == PIMDB_POT_DOUBLE_WELL) {
        s.ext_a = 4 * c.mass * c.ext_params[0];
        s.ext_b = c.ext_params[1] * c.ext_params[1];
        s.ext_c = c.mass * c.ext_params[0];
    } else if (c.ext_kind == PIMDB_POT_COSINE) {
        const double k = 2 * 3.14159265358979323846 / c.size;
        s.ext_a = -c.ext_params[0] * k;
        s.ext_b = k;
        s.ext_c = c.ext_params[1];
    }
    s.int_kind = c.int_kind;
    if (c.int_kind == PIMDB_POT_HARMONIC) s.int_a = c.mass * c.int_params[0] * c.int_params[0];
    else if (c.int_kind == PIMDB_POT_DIPOLE) s.int_a = c.int_params[0];
    s.seed = c.seed;
    s.replica = c.replica;
}

// Reference normal-mode rows (src/normal_modes.cpp:48-79), bit for bit.
void pimdb::nm_tables(int P, double omega_p, double mass, double dt, std::vector<double>& C,
                      std::vector<double>& T, std::vector<double>& rot) {
    const double pi = 3.14159265358979323846;
    C.assign((size_t)P * P, 0.0);
    T.assign((size_t)P * P, 0.0);
    rot.assign((size_t)P * 4, 0.0);
    for (int k = 0; k < P; ++k) {
        double* row = &C[(size_t)k * P];
        const double fund = 2 * pi / P * k;
        if (k == 0) {
            const double pref = 1 / std::sqrt((double)P);
            for (int i = 0; i < P; ++i) row[i] = pref;
        } else if (k < 0.5 * P) {
            const double pref = std::sqrt(2.0 / P);
            for (int i = 0; i < P; ++i) row[i] = pref * std::cos(fund * i);
        } else if (k == 0.5 * P) {
            const double pref = 1 / std::sqrt((double)P);
            for (int i = 0; i < P; ++i) row[i] = pref * (i % 2 == 0 ? 1.0 : -1.0);
        } else {
            const double pref = std::sqrt(2.0 / P);
            for (int i = 0; i < P; ++i) row[i] = -pref * std::sin(fund * i);
        }
        // normal_modes_propagator.cpp:13-16
        const double freq = 2 * omega_p * std::sin(k * pi / P);
        rot[4 * k] = std::cos(freq * dt);
        rot[4 * k + 1] = std::sin(freq * dt);
        rot[4 * k + 2] = mass * freq;
        // sin / (m omega_k) once here (IEEE division, as on the device)
        // instead of an FP64 division per mode and step (0 for the centroid,
        // which takes the free-particle branch)
        rot[4 * k + 3] = freq != 0.0 ? rot[4 * k + 1] / rot[4 * k + 2] : 0.0;
    }
    for (int j = 0; j < P; ++j) {
        double* row = &T[(size_t)j * P];
        const double fund = 2 * pi / P * j;
        const double pref = std::sqrt(2.0 / P);
        row[0] = 1 / std::sqrt((double)P);
        for (int i = 1; i < 0.5 * P; ++i) row[i] = pref * std::cos(fund * i);
        if (P % 2 == 0) row[P / 2] = 1 / std::sqrt((double)P) * (j % 2 == 0 ? 1.0 : -1.0);
        for (int i = (int)std::ceil(0.5 * (P + 1)); i < P; ++i) row[i] = -pref * std::sin(fund * i);
    }
}

static void free_handle(pimdb_handle* h) {
    double* bufs[] = {h->s.x,   h->s.p,   h->s.f,   h->s.fphys, h->s.fx,   h->s.E,        h->s.V,
                      h->s.Vb,  h->s.scal, h->s.Vh, h->s.Vbh,  h->s.yf,   h->s.yb,       h->s.Wf,
                      h->s.Wb,  h->s.Et, h->s.rowR, h->s.rowC, h->d_C,  h->d_T,    h->d_rot,      h->d_red[0],
                      h->d_red[1], h->d_stage, h->d_part, h->s.Vp, h->s.epart, h->d_obs};
    for (double* b : bufs)
        if (b) cudaFree(b);
    if (h->d_err) cudaFree(h->d_err);
    if (h->s.xflags) cudaFree(h->s.xflags);
    if (h->d_cmpart) cudaFree(h->d_cmpart);
    if (h->d_bar) cudaFree(h->d_bar);
    if (h->d_tw) cudaFree(h->d_tw);
    if (h->d_modes) cudaFree(h->d_modes);
    if (h->d_cells) cudaFree(h->d_cells);
    if (h->d_nh) cudaFree(h->d_nh);
    if (h->d_rng) cudaFree(h->d_rng);
    if (h->h_err) cudaFreeHost(h->h_err);
    if (h->d_ysol) cudaFree(h->d_ysol);
    if (h->d_ework) cudaFree(h->d_ework);
    if (h->d_gflags) cudaFree(h->d_gflags);
    if (h->d_noise) cudaFree(h->d_noise);
    if (h->d_pnm) cudaFree(h->d_pnm);
    if (h->d_step) cudaFree(h->d_step);
    drop_graphs(h);
    if (h->fork_ev) cudaEventDestroy(h->fork_ev);
    if (h->join_ev) cudaEventDestroy(h->join_ev);
    if (h->side) cudaStreamDestroy(h->side);
    if (h->ev0) cudaEventDestroy(h->ev0);
    if (h->ev1) cudaEventDestroy(h->ev1);
    if (h->own_stream && h->stream) cudaStreamDestroy(h->stream);
    delete h;
}

extern "C" int pimdb_create(const pimdb_config* cfg, void* cuda_stream, pimdb_handle** out) {
    if (!cfg || !out) return fail(nullptr, PIMDB_ERR_ARG, "NULL argument");
    *out = nullptr;
    const std::string why = validate_config(*cfg);
    if (!why.empty()) return fail(nullptr, PIMDB_ERR_CONFIG, why);
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
        cudaGetLastError();
        return fail(nullptr, PIMDB_ERR_NO_DEVICE, "no CUDA device visible");
    }
    pimdb_handle* h = new (std::nothrow) pimdb_handle();
    if (!h) return fail(nullptr, PIMDB_ERR_ARG, "out of host memory");
    h->cfg = *cfg;
    const pimdb_config& c = h->cfg;
    h->D = c.ndim;
    Sys& s = h->s;
    sys_params_from_config(c, s);

    auto alloc = [&](double** p, size_t n) -> cudaError_t {
        cudaError_t e = cudaMalloc((void**)p, std::max<size_t>(n, 1) * sizeof(double));
        if (e == cudaSuccess) e = cudaMemset(*p, 0, std::max<size_t>(n, 1) * sizeof(double));
        return e;
    };
    const size_t nstate = (size_t)s.P * h->D * s.ld;
    const int nred = std::max(cart_update_blocks(s, h->D), nm_blocks(s, h->D));
    cudaError_t e = cudaSuccess;
    if (cuda_stream) {
        h->stream = (cudaStream_t)cuda_stream;
    } else {
        e = cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking);
        h->own_stream = (e == cudaSuccess);
    }
    if (e == cudaSuccess) e = alloc(&s.x, nstate);
    if (e == cudaSuccess) e = alloc(&s.p, nstate);
    if (e == cudaSuccess) e = alloc(&s.f, nstate);
    if (e == cudaSuccess) e = alloc(&s.fphys, nstate);
    if (e == cudaSuccess) e = alloc(&s.fx, (size_t)2 * h->D * s.ld);
    if (e == cudaSuccess) e = alloc(&s.E, s.bosonic ? (size_t)s.N * (s.N + 1) / 2 : 1);
    if (e == cudaSuccess) e = alloc(&s.V, (size_t)s.N + 1);
    if (e == cudaSuccess) e = alloc(&s.Vb, (size_t)s.N + 1);
    if (e == cudaSuccess) e = alloc(&s.scal, 4);
    const size_t ntri = s.bosonic ? (size_t)s.N * (s.N + 1) / 2 : 1;
    if (e == cudaSuccess) e = alloc(&s.Vh, (size_t)s.N + 1);
    if (e == cudaSuccess) e = alloc(&s.Vbh, (size_t)s.N + 1);
    if (e == cudaSuccess) e = alloc(&s.yf, (size_t)s.N + 1);
    if (e == cudaSuccess) e = alloc(&s.yb, (size_t)s.N + 1);
    if (e == cudaSuccess) e = alloc(&s.Wf, ntri);
    if (e == cudaSuccess) e = alloc(&s.Wb, ntri);
    if (e == cudaSuccess) e = alloc(&s.Et, ntri);
    if (e == cudaSuccess) e = alloc(&s.rowR, (size_t)s.N);
    if (e == cudaSuccess) e = alloc(&s.rowC, (size_t)s.N);
    if (e == cudaSuccess && s.bosonic) {
        // no previous exchange result yet: NaN (0xff bytes) stops the first extrapolation
        e = cudaMalloc((void**)&s.Vp, 2 * ((size_t)s.N + 1) * sizeof(double));
        if (e == cudaSuccess) e = cudaMemset(s.Vp, 0xff, 2 * ((size_t)s.N + 1) * sizeof(double));
    }
    if (e == cudaSuccess && s.bosonic) e = alloc(&s.epart, kEstimatorDoubles);
    if (e == cudaSuccess && s.bosonic && exchange_energy_doubles(s, h->D) > 0)
        e = alloc(&h->d_ework, exchange_energy_doubles(s, h->D));
    if (e == cudaSuccess && s.bosonic && exchange_grid_doubles(s) > 0) {
        e = alloc(&h->d_ysol, exchange_grid_doubles(s));
        if (e == cudaSuccess) e = cudaMalloc((void**)&h->d_gflags, exchange_grid_flags(s) * sizeof(unsigned));
        if (e == cudaSuccess) e = cudaMemset(h->d_gflags, 0, exchange_grid_flags(s) * sizeof(unsigned));
    }
    // Newton's-third-law pair tiles need P * ceil(N/32) * D * ld partial sums;
    // when these (not what else the buffer holds) and the task counters exceed
    // 512 MiB the all-pairs kernel (no partials) is used instead.
    if (e == cudaSuccess && (pair_slot_doubles(s, h->D) + 1) * sizeof(double) <= (512ull << 20))
        e = alloc(&h->d_part, pair_partial_doubles(s, h->D));
    if (e == cudaSuccess) e = cudaMalloc((void**)&h->d_step, sizeof(long long));
    h->cell_nc = cell_grid(s, h->D);
    if (e == cudaSuccess && h->cell_nc > 0) e = cudaMalloc(&h->d_cells, cell_buffer_bytes(s, h->D, h->cell_nc));
    h->factorial = s.bosonic && c.exchange == PIMDB_EXCHANGE_FACTORIAL;
    if (e == cudaSuccess && c.rng == PIMDB_RNG_RANMAR && c.thermostat == PIMDB_THERMO_LANGEVIN) {
        std::vector<RanMarsState> st((size_t)s.P);
        for (int b = 0; b < s.P; ++b) ranmars_seed((int)(c.seed + (unsigned long long)b), st[b]);
        e = cudaMalloc((void**)&h->d_rng, st.size() * sizeof(RanMarsState));
        if (e == cudaSuccess)
            e = cudaMemcpy(h->d_rng, st.data(), st.size() * sizeof(RanMarsState), cudaMemcpyHostToDevice);
        // [step parity][substep][bead][axis][ld], plus one row of padding
        if (e == cudaSuccess) e = alloc(&h->d_noise, ((size_t)4 * s.P * h->D + 1) * s.ld);
        s.noise = h->d_noise;
    }
    // xflags: [0],[1] exact fallback used (forward, backward); [2] completion
    // counter; [3] next evaluation needs a fresh FP32 estimate; [4],[5] the
    // forward / backward solve asked for one; [6] retry pending; [7] the
    // estimate was reused; [kExchRetryCount] evaluations redone from a fresh
    // estimate after the reused one failed.
    if (e == cudaSuccess) e = cudaMalloc((void**)&s.xflags, 16 * sizeof(int));
    if (e == cudaSuccess) e = cudaMemset(s.xflags, 0, 16 * sizeof(int));
    const int one = 1;
    if (e == cudaSuccess) e = cudaMemcpy(s.xflags + 3, &one, sizeof(int), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = alloc(&h->d_red[0], com_doubles(nred));
    if (e == cudaSuccess) e = alloc(&h->d_red[1], com_doubles(nred));
    // host-order staging for the state crossing the boundary: [3][P*N*D]
    if (e == cudaSuccess) e = alloc(&h->d_stage, (size_t)3 * s.P * s.N * h->D);
    if (e == cudaSuccess) e = cudaMallocHost((void**)&h->h_err, sizeof(int));
    if (e == cudaSuccess) e = cudaMalloc((void**)&h->d_err, sizeof(int));
    if (e == cudaSuccess) e = cudaMemset(h->d_err, 0, sizeof(int));
    // the exchange chain's stream: highest priority, so its (latency-bound,
    // few-block) kernels are dispatched between the waves of the pair forces
    int prio_least = 0, prio_greatest = 0;
    if (e == cudaSuccess) e = cudaDeviceGetStreamPriorityRange(&prio_least, &prio_greatest);
    if (e == cudaSuccess) e = cudaStreamCreateWithPriority(&h->side, cudaStreamNonBlocking, prio_greatest);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&h->fork_ev, cudaEventDisableTiming);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&h->join_ev, cudaEventDisableTiming);
    if (e == cudaSuccess) e = cudaEventCreate(&h->ev0);
    if (e == cudaSuccess) e = cudaEventCreate(&h->ev1);
    if (e == cudaSuccess && (c.propagator == PIMDB_PROP_NORMAL_MODES || c.nmthermostat)) {
        std::vector<double> C, T, rot;
        nm_tables(s.P, s.omega_p, s.mass, s.dt, C, T, rot);
        e = alloc(&h->d_C, C.size());
        if (e == cudaSuccess) e = alloc(&h->d_T, T.size());
        if (e == cudaSuccess) e = alloc(&h->d_rot, rot.size());
        if (e == cudaSuccess) e = cudaMemcpy(h->d_C, C.data(), C.size() * sizeof(double), cudaMemcpyHostToDevice);
        if (e == cudaSuccess) e = cudaMemcpy(h->d_T, T.data(), T.size() * sizeof(double), cudaMemcpyHostToDevice);
        if (e == cudaSuccess)
            e = cudaMemcpy(h->d_rot, rot.data(), rot.size() * sizeof(double), cudaMemcpyHostToDevice);
    }
    if (e == cudaSuccess && c.thermostat >= PIMDB_THERMO_NOSE_HOOVER) {
        // constructors of nose_hoover.cpp:9-33, :149-158, :196-206
        const int D = h->D, N = s.N, P = s.P;
        NHPar& q = h->nh;
        q.variant = c.thermostat - PIMDB_THERMO_NOSE_HOOVER;
        q.nchains = c.nchains;
        const double beta = 1.0 / (1.0 * c.temperature);
        q.thermo_beta = beta / P;
        q.Qi = 1.0 * 1.0 * beta / P;
        q.Q1 = q.variant == 0 ? D * N * q.Qi : (q.variant == 1 ? D * q.Qi : q.Qi);
        q.required = q.variant == 0 ? D * N / q.thermo_beta : (q.variant == 1 ? D / q.thermo_beta : 1 / q.thermo_beta);
        q.dt2 = 0.5 * c.dt;
        q.dt4 = 0.25 * c.dt;
        q.dt8 = 0.125 * c.dt;
        h->nh_chains = q.variant == 0 ? P : (q.variant == 1 ? (long long)P * N : (long long)P * N * D);
        const size_t m = (size_t)h->nh_chains * q.nchains;
        e = alloc(&h->d_nh, 3 * m);
        q.eta = h->d_nh;
        q.eta_dot = h->d_nh + m;
        q.eta_dd = h->d_nh + 2 * m;
        if (e == cudaSuccess && c.nmthermostat) e = alloc(&h->d_pnm, (size_t)P * D * s.ld);
    }
    if (e == cudaSuccess && c.propagator == PIMDB_PROP_NORMAL_MODES && c.nmthermostat &&
        c.thermostat == PIMDB_THERMO_LANGEVIN && nm_fused_fits(s, h->D)) {
        e = alloc(&h->d_cmpart, nm_fused_partials(s, h->D));
        if (e == cudaSuccess) e = cudaMalloc((void**)&h->d_bar, 2 * sizeof(unsigned));
        if (e == cudaSuccess) e = cudaMemset(h->d_bar, 0, 2 * sizeof(unsigned));
        h->fused_nm = (e == cudaSuccess);
    }
    // FFT twiddles exp(-2 pi i t/P), t < P/2, for the normal-mode transforms
    if (e == cudaSuccess && (c.propagator == PIMDB_PROP_NORMAL_MODES || c.nmthermostat) && s.P >= 2 &&
        (s.P & (s.P - 1)) == 0) {
        const int P = s.P;
        std::vector<double> tw((size_t)P);
        const double pi = 3.14159265358979323846;
        for (int t = 0; t < P / 2; ++t) {
            tw[2 * t] = std::cos(2 * pi * t / P);
            tw[2 * t + 1] = -std::sin(2 * pi * t / P);
        }
        e = alloc(&h->d_tw, (size_t)P);
        if (e == cudaSuccess) e = cudaMemcpy(h->d_tw, tw.data(), (size_t)P * sizeof(double), cudaMemcpyHostToDevice);
        while ((1 << h->logP) < P) ++h->logP;
        if (e == cudaSuccess && (P == 32 || P == 64 || P == 128)) e = alloc(&h->d_modes, 2 * nm_mode_doubles(s, h->D));
    }
    cudaGetLastError();
    s.err = h->d_err;
    s.red = h->d_red[0];
    if (e != cudaSuccess) {
        std::string msg = std::string("allocation failed: ") + cudaGetErrorString(e);
        free_handle(h);
        return fail(nullptr, PIMDB_ERR_CUDA, msg);
    }
    *out = h;
    return PIMDB_OK;
}

extern "C" int pimdb_destroy(pimdb_handle* h) {
    if (!h) return PIMDB_ERR_ARG;
    if (h->stream) cudaStreamSynchronize(h->stream);
    free_handle(h);
    return PIMDB_OK;
}

static int check_err_word(pimdb_handle* h) {
    int err = 0;
    CUDA_TRY(h, cudaMemcpyAsync(&err, h->d_err, sizeof(int), cudaMemcpyDeviceToHost, h->stream));
    CUDA_TRY(h, cudaStreamSynchronize(h->stream));
    if (err) {
        CUDA_TRY(h, cudaMemsetAsync(h->d_err, 0, sizeof(int), h->stream));
        if (err & ERRB_NONFINITE_VB)
            return fail(h, PIMDB_ERR_NONFINITE_VB, "Invalid sig_denom in bosonic exchange potential");
        if (err & ERRB_TIMEOUT) return fail(h, PIMDB_ERR_TIMEOUT, "device wait timed out");
        return fail(h, PIMDB_ERR_BOUNDS, "device index check failed");
    }
    return PIMDB_OK;
}

// The device address of page-locked host memory (registered or allocated
// with the CUDA runtime), or null for any other pointer.  Kernels read and
// write such memory directly (over NVLink-C2C on Grace systems), which
// replaces a copy engine transfer plus a staging pass.
static void* pinned_view(const void* host) {
    if (!host) return nullptr;
    cudaPointerAttributes at{};
    if (cudaPointerGetAttributes(&at, host) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    return at.type == cudaMemoryTypeHost ? at.devicePointer : nullptr;
}

// The state kernels on device-accessible arrays (device memory, or the
// device views of page-locked host arrays).
static void state_in_launch(pimdb_handle* h, const double* sx, const double* sp) {
    h->modes_valid = false;
    launch(h, PIMDB_K_CART_UPDATE, [&] { launch_state_in(h->s, h->D, sx, sp, h->stream); });
    h->com_pending = false;
}
static void state_out_launch(pimdb_handle* h, double* ox, double* op, double* of) {
    if (ox || op || of) launch(h, PIMDB_K_CART_UPDATE, [&] { launch_state_out(h->s, h->D, ox, op, of, h->stream); });
}

// The state in, enqueued: one kernel (pack, zero the forces), reading
// page-locked host arrays directly or the staging buffer after a copy.
static int enqueue_state_in(pimdb_handle* h, const double* x, const double* p, cudaMemcpyKind kind) {
    if (h && x) ++h->xgen;
    complete_pending(h);
    const Sys& s = h->s;
    const size_t n = (size_t)s.P * s.N * h->D;
    const double* sx = x;
    const double* sp = p;
    if (kind == cudaMemcpyHostToDevice) {
        const double* vx = static_cast<const double*>(pinned_view(x));
        const double* vp = static_cast<const double*>(pinned_view(p));
        sx = x ? (vx ? vx : h->d_stage) : nullptr;
        sp = p ? (vp ? vp : h->d_stage + n) : nullptr;
        if (x && !vx) CUDA_TRY(h, cudaMemcpyAsync(h->d_stage, x, n * sizeof(double), kind, h->stream));
        if (p && !vp) CUDA_TRY(h, cudaMemcpyAsync(h->d_stage + n, p, n * sizeof(double), kind, h->stream));
    }
    state_in_launch(h, sx, sp);
    CUDA_TRY(h, cudaGetLastError());
    return PIMDB_OK;
}

// The state out, enqueued: the deferred tail of the last step, then one
// unpack kernel writing page-locked host arrays directly, or the staging
// buffer followed by a copy per array.
static int enqueue_state_out(pimdb_handle* h, double* x, double* p, double* f, cudaMemcpyKind kind) {
    complete_pending(h);
    const Sys& s = h->s;
    const size_t n = (size_t)s.P * s.N * h->D;
    double* dst[3] = {x, p, f};
    double* out[3] = {x, p, f};  // what the kernel writes
    bool copy[3] = {false, false, false};
    for (int k = 0; k < 3; ++k) {
        if (!dst[k] || kind != cudaMemcpyDeviceToHost) continue;
        double* v = static_cast<double*>(pinned_view(dst[k]));
        copy[k] = v == nullptr;
        out[k] = v ? v : h->d_stage + k * n;
    }
    state_out_launch(h, out[0], out[1], out[2]);
    for (int k = 0; k < 3; ++k)
        if (copy[k]) CUDA_TRY(h, cudaMemcpyAsync(dst[k], out[k], n * sizeof(double), kind, h->stream));
    CUDA_TRY(h, cudaGetLastError());
    return PIMDB_OK;
}

static int set_state_impl(pimdb_handle* h, const double* x, const double* p, cudaMemcpyKind kind) {
    if (!h) return PIMDB_ERR_ARG;
    const int st = enqueue_state_in(h, x, p, kind);
    if (st != PIMDB_OK) return st;
    CUDA_TRY(h, cudaStreamSynchronize(h->stream));
    return PIMDB_OK;
}

extern "C" int pimdb_set_state(pimdb_handle* h, const double* x, const double* p) {
    return set_state_impl(h, x, p, cudaMemcpyHostToDevice);
}
extern "C" int pimdb_set_state_device(pimdb_handle* h, const double* x, const double* p) {
    return set_state_impl(h, x, p, cudaMemcpyDeviceToDevice);
}

static int get_state_impl(pimdb_handle* h, double* x, double* p, double* f, cudaMemcpyKind kind) {
    if (!h) return PIMDB_ERR_ARG;
    const int st = enqueue_state_out(h, x, p, f, kind);
    if (st != PIMDB_OK) return st;
    CUDA_TRY(h, cudaStreamSynchronize(h->stream));
    return PIMDB_OK;
}

extern "C" int pimdb_get_state(pimdb_handle* h, double* x, double* p, double* f) {
    return get_state_impl(h, x, p, f, cudaMemcpyDeviceToHost);
}
extern "C" int pimdb_get_state_device(pimdb_handle* h, double* x, double* p, double* f) {
    return get_state_impl(h, x, p, f, cudaMemcpyDeviceToDevice);
}

extern "C" int pimdb_set_step(pimdb_handle* h, long long step) {
    if (!h) return PIMDB_ERR_ARG;
    h->step = step;
    h->dstep_valid = false;
    return PIMDB_OK;
}
extern "C" int pimdb_get_step(pimdb_handle* h, long long* step) {
    if (!h || !step) return PIMDB_ERR_ARG;
    *step = h->step;
    return PIMDB_OK;
}

// The exchange on beads 1 and P in two parts.  exchange_front: everything
// up to the forces (Feldman-Hirshberg: cycle energies and the V / V_backwards
// recursions, which give V_B; factorial: nothing).  exchange_forces: the
// exterior spring forces into fx, also added into f with `accumulate`
// (factorial: the whole exchange).
static void exchange_front(pimdb_handle* h, cudaStream_t st) {
    const Sys& s = h->s;
    if (h->factorial) return;
    int est = 0;
    launch(h, PIMDB_K_EXCH_ENERGIES, [&] { est = launch_exchange_energies(s, h->D, st, h->d_ework); },
           h->d_ework && s.eflat ? 3 : 1);
    const int ex = h->opt_exact_exchange;
    int nk = 0;
    launch(h, PIMDB_K_EXCH_RECURSIONS,
           [&] { nk = launch_exchange_recursions(s, ex, st, h->d_ysol, h->d_gflags, est); }, 0);
    h->launches += nk;
}
static void exchange_forces(pimdb_handle* h, int accumulate, cudaStream_t st) {
    const Sys& s = h->s;
    if (h->factorial)
        launch(h, PIMDB_K_EXCH_FORCES, [&] { launch_factorial(s, h->D, accumulate, st); });
    else
        launch(h, PIMDB_K_EXCH_FORCES, [&] { launch_exchange_forces_mode(s, h->D, accumulate, st); });
}
// All four scalars after exchange_front (and, for the factorial sum, with or
// without exchange_forces before).
static void exchange_scalars(pimdb_handle* h, bool forces_done, cudaStream_t st) {
    if (h->factorial) {
        if (!forces_done) exchange_forces(h, 0, st);
        return;
    }
    launch(h, PIMDB_K_EXCH_ESTIMATORS, [&] { launch_exchange_estimators(h->s, st); });
}

// Simulation::updateForces for all beads.
static void enqueue_forces(pimdb_handle* h) {
    const Sys& s = h->s;
    const bool nm = h->cfg.propagator == PIMDB_PROP_NORMAL_MODES;
    // exchange chain on the side stream when not profiling (profiling times
    // every launch on the main stream)
    const bool fork = s.bosonic && !h->profile;
    cudaStream_t xs = fork ? h->side : h->stream;
    if (fork) {
        cudaEventRecord(h->fork_ev, h->stream);
        cudaStreamWaitEvent(h->side, h->fork_ev, 0);
    }
    const int mixed = h->cfg.precision == PIMDB_MIXED;
    const bool cells = h->d_cells && (h->opt_cells == 1 || (h->opt_cells < 0 && s.N >= 512));
    const bool tiles = !cells && h->d_part && h->opt_newton3;
    // with the tile or cell paths the exchange forces go to fx on the side
    // stream and the finishing kernel adds them: off the critical path
    const bool fx_in_finish = s.bosonic && (cells || tiles);
    // With the pair tiles and the exchange on two streams, the tiles leave
    // SMs to the exchange's one-block passes (estimate, solve), whose
    // sequential chains would otherwise share the FP64 pipes with them.
    h->s.reserve_sms =
        fork && tiles ? (h->opt_reserved_sms >= 0 ? h->opt_reserved_sms : exchange_reserved_sms(s)) : 0;
    if (s.bosonic) {
        exchange_front(h, xs);
        if (fx_in_finish) exchange_forces(h, 0, xs);
    }
    if (fork) cudaEventRecord(h->join_ev, h->side);
    cudaEvent_t before_finish = fork && fx_in_finish ? h->join_ev : nullptr;
    if (cells) {
        launch(h, PIMDB_K_BEAD_FORCES, [&] {
            launch_pair_cells_and_finish(s, h->D, h->cell_nc, mixed, nm ? 1 : 0, h->d_cells, before_finish,
                                         fx_in_finish, h->stream);
        }, 3);
    } else if (tiles) {
        launch(
            h, PIMDB_K_BEAD_FORCES,
            [&] {
                launch_pair_tiles_and_finish(s, h->D, mixed, nm ? 1 : 0, h->d_part, before_finish, fx_in_finish,
                                             h->stream);
            },
            pair_tile_kernels(s, mixed));
    } else {
        launch(h, PIMDB_K_BEAD_FORCES, [&] { launch_bead_forces(s, h->D, mixed, nm ? 1 : 0, h->stream); });
    }
    if (fork && !fx_in_finish) cudaStreamWaitEvent(h->stream, h->join_ev, 0);
    if (s.bosonic && !fx_in_finish) exchange_forces(h, 1, h->stream);
}

extern "C" int pimdb_compute_forces(pimdb_handle* h) {
    if (!h) return PIMDB_ERR_ARG;
    complete_pending(h);
    enqueue_forces(h);
    CUDA_TRY(h, cudaGetLastError());
    return check_err_word(h);
}

// Momentum kernels with the COM bookkeeping: a kernel that applies the
// pending correction reads buffer red_last and writes new partials into the
// other buffer.
static void cart(pimdb_handle* h, int flags, int substep, int kick_nm) {
    h->modes_valid = false;
    const int rin = h->red_last, rout = 1 - h->red_last;
    if (!h->com_pending) flags &= ~SF_COM_APPLY;
    launch(h, PIMDB_K_CART_UPDATE, [&] {
        launch_cart_update(h->s, h->D, flags, h->d_red[rin], h->nred_last, h->d_red[rout], step_ref(h, h->step), substep,
                           kick_nm, h->stream);
    });
    if (flags & SF_COM_APPLY) h->com_pending = false;
    if (flags & SF_COM_PARTIAL) {
        h->red_last = rout;
        h->nred_last = cart_update_blocks(h->s, h->D);
        h->com_pending = true;
    }
}

static void nm_thermo(pimdb_handle* h, int flags, int substep) {
    h->modes_valid = false;
    const int rin = h->red_last, rout = 1 - h->red_last;
    if (!h->com_pending) flags &= ~SF_COM_APPLY;
    launch(h, PIMDB_K_NM_THERMO, [&] {
        launch_nm_thermo(h->s, h->D, h->d_C, h->d_T, flags, h->d_red[rin], h->nred_last, h->d_red[rout],
                         step_ref(h, h->step), substep, h->stream);
    });
    if (flags & SF_COM_APPLY) h->com_pending = false;
    if (flags & SF_COM_PARTIAL) {
        h->red_last = rout;
        h->nred_last = nm_blocks(h->s, h->D);
        h->com_pending = true;
    }
}

// Applies the O-step of the configured thermostat (thermostat.cpp:15-19)
// followed, when fixcom, by the partial sums for the COM removal.
static void nose_hoover(pimdb_handle* h) {
    h->modes_valid = false;
    const bool nmc = h->cfg.nmthermostat != 0;
    launch(h, PIMDB_K_NM_THERMO, [&] {
        launch_nose_hoover(h->s, h->D, h->nh, nmc ? h->d_C : nullptr, nmc ? h->d_T : nullptr, h->d_pnm, h->stream);
    }, nmc ? 3 : 1);
}

// RanMars parity noise: both O-steps' normals of MD step `step`, from the
// streams' current positions (the step before's stay in the other half).
static void draw_noise(pimdb_handle* h, long long step) {
    if (!h->d_noise) return;
    launch(h, PIMDB_K_CART_UPDATE, [&] {
        launch_ranmars_draw(h->s, h->D, h->d_rng, h->d_noise, step_ref(h, step), h->stream);
    });
}

static void thermostat_step(pimdb_handle* h, int substep) {
    const pimdb_config& c = h->cfg;
    const int part = c.fixcom ? SF_COM_PARTIAL : 0;
    if (c.thermostat >= PIMDB_THERMO_NOSE_HOOVER) {
        // the pending COM correction first, then the chains; partial sums
        // for the COM removal that follows (simulation.cpp:246-258)
        if (h->com_pending) cart(h, SF_COM_APPLY, substep, 0);
        nose_hoover(h);
        if (c.fixcom) cart(h, SF_COM_PARTIAL, substep, 0);
    } else if (c.thermostat == PIMDB_THERMO_LANGEVIN && c.nmthermostat) {
        nm_thermo(h, SF_COM_APPLY | part, substep);
    } else if (c.thermostat == PIMDB_THERMO_LANGEVIN) {
        cart(h, SF_COM_APPLY | SF_LANGEVIN | part, substep, 0);
    } else if (c.fixcom || h->com_pending) {
        cart(h, SF_COM_APPLY | part, substep, 0);
    }
}

static void enqueue_steps(pimdb_handle* h, int nsteps) {
    const pimdb_config& c = h->cfg;
    const bool nm = c.propagator == PIMDB_PROP_NORMAL_MODES;
    const bool cart_langevin = c.thermostat == PIMDB_THERMO_LANGEVIN && !c.nmthermostat;
    // The last momentum update of a step with the Cartesian Langevin
    // thermostat: B, O and, when another step follows, that step's first O in
    // the same pass (COM O2, COM O1 = COM after both: the removal is a linear
    // projection and O is affine).
    auto kick_langevin = [&](bool more, int kick_nm) {
        if (more) draw_noise(h, h->step + 1);
        cart(h, SF_KICK | SF_LANGEVIN | (more ? SF_LANGEVIN_NEXT : 0) | (c.fixcom ? SF_COM_PARTIAL : 0), 1, kick_nm);
    };
    bool head_done = false;  // this step's first O was part of the previous step's last pass
    for (int it = 0; it < nsteps; ++it) {
        const bool more = it + 1 < nsteps;
        // O, [COM] (inside the fused normal-mode kernel when that is used)
        if (!head_done) {
            draw_noise(h, h->step);
            if (!(nm && h->fused_nm)) thermostat_step(h, 0);
        }
        if (!nm) {
            // [COM], B, A (velocity_verlet.cpp:9-12)
            cart(h, SF_COM_APPLY | SF_KICK | SF_DRIFT, 0, 0);
            enqueue_forces(h);
            // B, then O (+ partials) when the thermostat is Cartesian Langevin
            if (cart_langevin) {
                kick_langevin(more, 0);
                head_done = more;
            } else {
                cart(h, SF_KICK, 1, 0);
                thermostat_step(h, 1);
            }
        } else if (h->fused_nm) {
            // tail of the previous step (if pending) and head of this one
            const int mode = (h->nm_tail_pending ? 1 : 0) | 2;
            const long long st = h->step;
            const size_t nmd = h->d_modes ? nm_mode_doubles(h->s, h->D) : 0;
            const NmModes mm{(double2*)h->d_modes, (double2*)(h->d_modes + nmd),
                             h->modes_valid && h->nm_tail_pending ? 1 : 0, false};
            launch(h, PIMDB_K_NM_PROPAGATE, [&] {
                cudaError_t e = launch_nm_fused(h->s, h->D, h->d_C, h->d_T, h->d_rot, h->d_cmpart, h->d_bar, mode,
                                                step_ref(h, st), c.fixcom,
                                                h->opt_fft ? (const double2*)h->d_tw : nullptr, h->logP, h->stream,
                                                h->d_modes ? &mm : nullptr);
                if (e != cudaSuccess) h->async_err = e;
            });
            h->modes_valid = h->d_modes != nullptr && mm.written;
            enqueue_forces(h);
            h->nm_tail_pending = true;
        } else {
            // [COM] + half-kick + free ring-polymer propagation
            h->modes_valid = false;
            const int rin = h->red_last;
            const int apply = h->com_pending ? 1 : 0;
            launch(h, PIMDB_K_NM_PROPAGATE, [&] {
                launch_nm_propagate(h->s, h->D, h->d_C, h->d_T, h->d_rot, apply, h->d_red[rin], h->nred_last,
                                    h->opt_fft ? (const double2*)h->d_tw : nullptr, h->stream);
            });
            h->com_pending = false;
            enqueue_forces(h);
            if (cart_langevin) {
                kick_langevin(more, 1);
                head_done = more;
            } else {
                cart(h, SF_KICK, 1, 1);
                thermostat_step(h, 1);
            }
        }
        h->step += 1;
    }
}

// Work of the last step deferred until the host needs the state: the tail
// of the fused normal-mode kernel (kick, O-step, COM removal) and a pending
// COM correction.  The next step absorbs both when it comes first, so a
// run of pimdb_step calls pays for one fused launch per step.
static void complete_pending(pimdb_handle* h) {
    if (h->nm_tail_pending || h->com_pending) h->modes_valid = false;  // the tail changes p
    if (h->nm_tail_pending) {
        const long long st = h->step;
        launch(h, PIMDB_K_NM_PROPAGATE, [&] {
            cudaError_t e = launch_nm_fused(h->s, h->D, h->d_C, h->d_T, h->d_rot, h->d_cmpart, h->d_bar, 1,
                                            step_ref(h, st), h->cfg.fixcom,
                                            h->opt_fft ? (const double2*)h->d_tw : nullptr, h->logP, h->stream);
            if (e != cudaSuccess) h->async_err = e;
        });
        h->nm_tail_pending = false;
    }
    if (h->com_pending) cart(h, SF_COM_APPLY, 0, 0);
}

// `nsteps` steps as one CUDA graph (captured on first use for this step
// state, then replayed).  Returns false when graphs cannot be used here;
// the caller then enqueues the steps directly.
static bool graph_steps(pimdb_handle* h, int nsteps) {
    if (!h->opt_graph || h->graph_broken || h->profile || !h->warm || nsteps < 1) return false;
    const pimdb_handle::StepState before{h->red_last, h->nred_last, h->com_pending, h->nm_tail_pending,
                                         h->modes_valid};
    const auto key = std::make_pair(nsteps, before);
    auto it = h->graphs.find(key);
    if (it == h->graphs.end()) {
        pimdb_handle::StepGraph g;
        const long long step0 = h->step, launches0 = h->launches;
        cudaGraph_t graph = nullptr;
        if (cudaStreamBeginCapture(h->stream, cudaStreamCaptureModeThreadLocal) != cudaSuccess) {
            cudaGetLastError();
            h->graph_broken = true;
            return false;
        }
        h->capturing = true;
        h->graph_base = step0;
        enqueue_steps(h, nsteps);
        launch_step_advance(h->d_step, nsteps, h->stream);
        h->capturing = false;
        cudaError_t e = cudaStreamEndCapture(h->stream, &graph);
        // kernel nodes keep the priority of the stream they were captured on
        // (the exchange chain's stream is the higher one)
        if (e == cudaSuccess && h->async_err == cudaSuccess)
            e = cudaGraphInstantiateWithFlags(&g.exec, graph, cudaGraphInstantiateFlagUseNodePriority);
        if (graph) cudaGraphDestroy(graph);
        g.after = {h->red_last, h->nred_last, h->com_pending, h->nm_tail_pending, h->modes_valid};
        g.kernels = h->launches - launches0 + 1;
        // the capture only recorded the work: restore the host state
        h->step = step0;
        h->launches = launches0;
        h->red_last = before.red_last;
        h->nred_last = before.nred_last;
        h->com_pending = before.com_pending;
        h->nm_tail_pending = before.nm_tail_pending;
        h->modes_valid = before.modes_valid;
        if (e != cudaSuccess || h->async_err != cudaSuccess) {
            cudaGetLastError();
            h->async_err = cudaSuccess;
            if (g.exec) cudaGraphExecDestroy(g.exec);
            h->graph_broken = true;
            return false;
        }
        it = h->graphs.emplace(key, g).first;
    }
    if (!h->dstep_valid) {
        if (cudaStreamSynchronize(h->stream) != cudaSuccess ||
            cudaMemcpy(h->d_step, &h->step, sizeof(long long), cudaMemcpyHostToDevice) != cudaSuccess) {
            h->async_err = cudaGetLastError();
            return true;
        }
        h->dstep_valid = true;
    }
    const cudaError_t e = cudaGraphLaunch(it->second.exec, h->stream);
    if (e != cudaSuccess) h->async_err = e;
    h->step += nsteps;
    h->launches += it->second.kernels;
    const pimdb_handle::StepState& a = it->second.after;
    h->red_last = a.red_last;
    h->nred_last = a.nred_last;
    h->com_pending = a.com_pending;
    h->nm_tail_pending = a.nm_tail_pending;
    h->modes_valid = a.modes_valid;
    return true;
}

extern "C" int pimdb_step_async(pimdb_handle* h, int nsteps) {
    if (!h || nsteps < 0) return PIMDB_ERR_ARG;
    if (nsteps > 0) ++h->xgen;
    if (!graph_steps(h, nsteps)) {
        enqueue_steps(h, nsteps);
        h->dstep_valid = false;
        h->warm = nsteps > 0;
    }
    if (h->async_err != cudaSuccess) {
        const cudaError_t e = h->async_err;
        h->async_err = cudaSuccess;
        return fail(h, PIMDB_ERR_CUDA, std::string("kernel launch: ") + cudaGetErrorString(e));
    }
    CUDA_TRY(h, cudaGetLastError());
    return PIMDB_OK;
}

extern "C" int pimdb_step(pimdb_handle* h, int nsteps) {
    int st = pimdb_step_async(h, nsteps);
    if (st != PIMDB_OK) return st;
    return check_err_word(h);
}

// A whole pimdb_step_io call as one CUDA graph when every host array given
// is page-locked (the state kernels then read and write them directly):
// state in, the steps, the deferred tail, state out and the error word, with
// no host work between them.  Returns -1 when it does not apply (the caller
// enqueues the call), else the status of the launch.
static int graph_io(pimdb_handle* h, const double* xi, const double* pi, int nsteps, double* xo, double* po,
                    double* fo) {
    if (!h->opt_graph || h->graph_broken || h->profile || !h->warm || nsteps < 1) return -1;
    ++h->xgen;
    const void* host[5] = {xi, pi, xo, po, fo};
    pimdb_handle::IoKey key{};
    key.nsteps = nsteps;
    key.before = {h->red_last, h->nred_last, h->com_pending, h->nm_tail_pending, h->modes_valid};
    for (int k = 0; k < 5; ++k) {
        key.v[k] = host[k] ? pinned_view(host[k]) : nullptr;
        if (host[k] && !key.v[k]) return -1;
    }
    auto it = h->io_graphs.find(key);
    if (it == h->io_graphs.end()) {
        if (h->io_graphs.size() >= 8) {  // callers passing new arrays every time
            for (auto& kv : h->io_graphs)
                if (kv.second.exec) cudaGraphExecDestroy(kv.second.exec);
            h->io_graphs.clear();
        }
        pimdb_handle::StepGraph g;
        const pimdb_handle::StepState before = key.before;
        const long long step0 = h->step, launches0 = h->launches;
        cudaGraph_t graph = nullptr;
        if (cudaStreamBeginCapture(h->stream, cudaStreamCaptureModeThreadLocal) != cudaSuccess) {
            cudaGetLastError();
            h->graph_broken = true;
            return -1;
        }
        h->capturing = true;
        h->graph_base = step0;
        if (xi || pi) {
            complete_pending(h);
            state_in_launch(h, static_cast<const double*>(key.v[0]), static_cast<const double*>(key.v[1]));
        }
        enqueue_steps(h, nsteps);
        complete_pending(h);
        state_out_launch(h, (double*)key.v[2], (double*)key.v[3], (double*)key.v[4]);
        // last: every captured kernel reads the step index relative to the
        // device counter as it was when the graph started
        launch_step_advance(h->d_step, nsteps, h->stream);
        cudaMemcpyAsync(h->h_err, h->d_err, sizeof(int), cudaMemcpyDeviceToHost, h->stream);
        h->capturing = false;
        cudaError_t e = cudaStreamEndCapture(h->stream, &graph);
        if (e == cudaSuccess && h->async_err == cudaSuccess)
            e = cudaGraphInstantiateWithFlags(&g.exec, graph, cudaGraphInstantiateFlagUseNodePriority);
        if (graph) cudaGraphDestroy(graph);
        g.after = {h->red_last, h->nred_last, h->com_pending, h->nm_tail_pending, h->modes_valid};
        g.kernels = h->launches - launches0 + 1;
        // the capture only recorded the work: restore the host state
        h->step = step0;
        h->launches = launches0;
        h->red_last = before.red_last;
        h->nred_last = before.nred_last;
        h->com_pending = before.com_pending;
        h->nm_tail_pending = before.nm_tail_pending;
        h->modes_valid = before.modes_valid;
        if (e != cudaSuccess || h->async_err != cudaSuccess) {
            cudaGetLastError();
            h->async_err = cudaSuccess;
            if (g.exec) cudaGraphExecDestroy(g.exec);
            h->graph_broken = true;
            return -1;
        }
        it = h->io_graphs.emplace(key, g).first;
    }
    if (!h->dstep_valid) {
        CUDA_TRY(h, cudaStreamSynchronize(h->stream));
        CUDA_TRY(h, cudaMemcpy(h->d_step, &h->step, sizeof(long long), cudaMemcpyHostToDevice));
        h->dstep_valid = true;
    }
    CUDA_TRY(h, cudaGraphLaunch(it->second.exec, h->stream));
    h->step += nsteps;
    h->launches += it->second.kernels;
    const pimdb_handle::StepState& a = it->second.after;
    h->red_last = a.red_last;
    h->nred_last = a.nred_last;
    h->com_pending = a.com_pending;
    h->nm_tail_pending = a.nm_tail_pending;
    h->modes_valid = a.modes_valid;
    return PIMDB_OK;
}

extern "C" int pimdb_step_io(pimdb_handle* h, const double* x_in, const double* p_in, int nsteps, double* x_out,
                             double* p_out, double* f_out) {
    if (!h || nsteps < 0) return PIMDB_ERR_ARG;
    const int gio = graph_io(h, x_in, p_in, nsteps, x_out, p_out, f_out);
    if (gio > 0) return gio;
    if (gio == 0) {
        CUDA_TRY(h, cudaStreamSynchronize(h->stream));
        return *h->h_err ? check_err_word(h) : PIMDB_OK;
    }
    int st = PIMDB_OK;
    if (x_in || p_in) st = enqueue_state_in(h, x_in, p_in, cudaMemcpyHostToDevice);
    if (st == PIMDB_OK && nsteps > 0) st = pimdb_step_async(h, nsteps);
    if (st == PIMDB_OK) st = enqueue_state_out(h, x_out, p_out, f_out, cudaMemcpyDeviceToHost);
    if (st != PIMDB_OK) {
        cudaStreamSynchronize(h->stream);
        return st;
    }
    // the error word travels with the outputs: one synchronisation in all
    CUDA_TRY(h, cudaMemcpyAsync(h->h_err, h->d_err, sizeof(int), cudaMemcpyDeviceToHost, h->stream));
    CUDA_TRY(h, cudaStreamSynchronize(h->stream));
    return *h->h_err ? check_err_word(h) : PIMDB_OK;
}

extern "C" int pimdb_synchronize(pimdb_handle* h) {
    if (!h) return PIMDB_ERR_ARG;
    CUDA_TRY(h, cudaGetLastError());
    return check_err_word(h);
}

extern "C" int pimdb_exchange(pimdb_handle* h, double* scalars, double* f_first, double* f_last) {
    if (!h) return PIMDB_ERR_ARG;
    complete_pending(h);
    const Sys& s = h->s;
    if (!s.bosonic) return fail(h, PIMDB_ERR_CONFIG, "pimdb_exchange needs a bosonic configuration with nbeads > 1");
    exchange_front(h, h->stream);
    exchange_forces(h, 0, h->stream);
    exchange_scalars(h, true, h->stream);
    CUDA_TRY(h, cudaGetLastError());
    int st = check_err_word(h);
    if (st != PIMDB_OK) return st;
    if (scalars) CUDA_TRY(h, cudaMemcpy(scalars, s.scal, 4 * sizeof(double), cudaMemcpyDeviceToHost));
    const int D = h->D;
    std::vector<double> fx((size_t)2 * D * s.ld);
    if (f_first || f_last) {
        CUDA_TRY(h, cudaMemcpy(fx.data(), s.fx, fx.size() * sizeof(double), cudaMemcpyDeviceToHost));
        for (int side = 0; side < 2; ++side) {
            double* out = side == 0 ? f_first : f_last;
            if (!out) continue;
            for (int i = 0; i < s.N; ++i)
                for (int a = 0; a < D; ++a) out[(size_t)i * D + a] = fx[((size_t)side * D + a) * s.ld + i];
        }
    }
    return PIMDB_OK;
}

static int fh_exchange_only(pimdb_handle* h, const char* what) {
    if (!h->s.bosonic || h->factorial)
        return fail(h, PIMDB_ERR_CONFIG,
                    std::string(what) + " needs the Feldman-Hirshberg exchange (bosonic, nbeads > 1)");
    return PIMDB_OK;
}

static int exchange_forward_current(pimdb_handle* h, const char* what) {
    if (h->fwd_gen != h->xgen)
        return fail(h, PIMDB_ERR_ARG,
                    std::string(what) + " needs pimdb_exchange_forward on the current coordinates first");
    return PIMDB_OK;
}

extern "C" int pimdb_exchange_retries(pimdb_handle* h, long long* count) {
    if (!h || !count) return PIMDB_ERR_ARG;
    *count = 0;
    if (!h->s.bosonic || h->factorial) return PIMDB_OK;
    int v = 0;
    CUDA_TRY(h, cudaMemcpyAsync(&v, h->s.xflags + kExchRetryCount, sizeof(int), cudaMemcpyDeviceToHost, h->stream));
    CUDA_TRY(h, cudaStreamSynchronize(h->stream));
    *count = v;
    return PIMDB_OK;
}

extern "C" int pimdb_exchange_fresh_estimates(pimdb_handle* h, long long* count) {
    if (!h || !count) return PIMDB_ERR_ARG;
    *count = 0;
    if (!h->s.bosonic || h->factorial) return PIMDB_OK;
    int v = 0;
    CUDA_TRY(h, cudaMemcpyAsync(&v, h->s.xflags + kExchFreshCount, sizeof(int), cudaMemcpyDeviceToHost, h->stream));
    CUDA_TRY(h, cudaStreamSynchronize(h->stream));
    *count = v;
    return PIMDB_OK;
}

extern "C" int pimdb_exchange_forward(pimdb_handle* h, double* VB) {
    if (!h) return PIMDB_ERR_ARG;
    int st = fh_exchange_only(h, "pimdb_exchange_forward");
    if (st != PIMDB_OK) return st;
    complete_pending(h);
    exchange_front(h, h->stream);
    CUDA_TRY(h, cudaGetLastError());
    st = check_err_word(h);
    if (st != PIMDB_OK) return st;
    h->fwd_gen = h->xgen;
    if (VB) CUDA_TRY(h, cudaMemcpy(VB, h->s.V + h->s.N, sizeof(double), cudaMemcpyDeviceToHost));
    return PIMDB_OK;
}

extern "C" int pimdb_exchange_adjoint(pimdb_handle* h, double vb_bar, double* x1_bar, double* xP_bar) {
    if (!h) return PIMDB_ERR_ARG;
    int st = fh_exchange_only(h, "pimdb_exchange_adjoint");
    if (st == PIMDB_OK) st = exchange_forward_current(h, "pimdb_exchange_adjoint");
    if (st != PIMDB_OK) return st;
    const Sys& s = h->s;
    const int D = h->D;
    launch(h, PIMDB_K_EXCH_FORCES, [&] { launch_exchange_adjoint(s, D, vb_bar, h->stream); });
    CUDA_TRY(h, cudaGetLastError());
    std::vector<double> fx((size_t)2 * D * s.ld);
    CUDA_TRY(h, cudaMemcpyAsync(fx.data(), s.fx, fx.size() * sizeof(double), cudaMemcpyDeviceToHost, h->stream));
    CUDA_TRY(h, cudaStreamSynchronize(h->stream));
    for (int side = 0; side < 2; ++side) {
        double* out = side == 0 ? x1_bar : xP_bar;
        if (!out) continue;
        for (int i = 0; i < s.N; ++i)
            for (int a = 0; a < D; ++a) out[(size_t)i * D + a] = fx[((size_t)side * D + a) * s.ld + i];
    }
    return PIMDB_OK;
}

extern "C" int pimdb_exchange_dbeta(pimdb_handle* h, double* dbeta) {
    if (!h || !dbeta) return fail(h, PIMDB_ERR_ARG, "NULL argument");
    int st = fh_exchange_only(h, "pimdb_exchange_dbeta");
    if (st == PIMDB_OK) st = exchange_forward_current(h, "pimdb_exchange_dbeta");
    if (st != PIMDB_OK) return st;
    exchange_scalars(h, false, h->stream);
    CUDA_TRY(h, cudaGetLastError());
    CUDA_TRY(h, cudaMemcpyAsync(dbeta, h->s.scal + 1, sizeof(double), cudaMemcpyDeviceToHost, h->stream));
    CUDA_TRY(h, cudaStreamSynchronize(h->stream));
    return PIMDB_OK;
}

// The exchange beside other kernels: begins on the side stream (the handle's
// stream when profiling, which times every launch there) ...
static cudaStream_t fork_exchange(pimdb_handle* h) {
    if (!h->s.bosonic || h->profile) return h->stream;
    cudaEventRecord(h->fork_ev, h->stream);
    cudaStreamWaitEvent(h->side, h->fork_ev, 0);
    return h->side;
}
// ... and what follows on the handle's stream waits for it.
static void join_exchange(pimdb_handle* h, cudaStream_t xs) {
    if (xs == h->stream) return;
    cudaEventRecord(h->join_ev, xs);
    cudaStreamWaitEvent(h->stream, h->join_ev, 0);
}

// The per-block terms (`per` doubles per bead and block of energy_blocks) and
// the estimators' tile energies, kept from the first call on.
static int obs_work(pimdb_handle* h, double** part, double** tiles) {
    const Sys& s = h->s;
    const size_t n = (size_t)s.P * energy_blocks(s) * 7;
    if (!h->d_obs)
        CUDA_TRY(h, cudaMalloc((void**)&h->d_obs, (n + (h->d_part ? energy_tile_doubles(s) : 0)) * sizeof(double)));
    *part = h->d_obs;
    *tiles = h->d_obs + n;
    return PIMDB_OK;
}
// Kernels of an energy evaluation: the tiles, when there are pairs and room
// for their partial sums, and the per-bead terms.
static int tile_launches(const pimdb_handle* h) {
    return h->d_part && h->s.int_kind != PIMDB_POT_FREE && h->s.cutoff != 0.0 ? 2 : 1;
}
// SMs the tiles leave to an exchange on another stream (as enqueue_forces).
static void reserve_for_exchange(pimdb_handle* h, bool beside) {
    h->s.reserve_sms =
        beside && h->d_part ? (h->opt_reserved_sms >= 0 ? h->opt_reserved_sms : exchange_reserved_sms(h->s)) : 0;
}

extern "C" int pimdb_potential_energy(pimdb_handle* h, double* terms) {
    if (!h || !terms) return fail(h, PIMDB_ERR_ARG, "NULL argument");
    complete_pending(h);
    const Sys& s = h->s;
    const int nb = energy_blocks(s);
    const size_t n = (size_t)s.P * nb * 3;
    double *part = nullptr, *tiles = nullptr;
    const int ws = obs_work(h, &part, &tiles);
    if (ws != PIMDB_OK) return ws;
    const cudaStream_t xs = fork_exchange(h);
    reserve_for_exchange(h, xs != h->stream);
    if (s.bosonic) {
        exchange_front(h, xs);
        if (h->factorial) exchange_scalars(h, false, xs);
    }
    launch(h, PIMDB_K_BEAD_FORCES, [&] { launch_energy_terms(s, h->D, part, tiles, h->d_part, h->stream); },
           tile_launches(h));
    join_exchange(h, xs);
    std::vector<double> hp(n);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpyAsync(hp.data(), part, n * sizeof(double), cudaMemcpyDeviceToHost, h->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(h->stream);
    if (e != cudaSuccess) return fail(h, PIMDB_ERR_CUDA, cudaGetErrorString(e));
    const int st = check_err_word(h);
    if (st != PIMDB_OK) return st;
    for (int k = 0; k < 3; ++k) {
        double t = 0.0;
        for (size_t q = 0; q < (size_t)s.P * nb; ++q) t += hp[q * 3 + k];
        terms[k] = t;
    }
    terms[3] = 0.0;
    if (s.bosonic) CUDA_TRY(h, cudaMemcpy(&terms[3], s.scal, sizeof(double), cudaMemcpyDeviceToHost));
    return PIMDB_OK;
}

extern "C" int pimdb_compute_observables(pimdb_handle* h, pimdb_observables* out) {
    if (!h || !out) return fail(h, PIMDB_ERR_ARG, "NULL argument");
    complete_pending(h);
    const Sys& s = h->s;
    const int D = h->D, P = s.P, N = s.N;
    const int nb = energy_blocks(s);
    const size_t n = (size_t)P * nb * 7;
    double *part = nullptr, *tiles = nullptr;
    const int ws = obs_work(h, &part, &tiles);
    if (ws != PIMDB_OK) return ws;
    const cudaStream_t xs = fork_exchange(h);
    reserve_for_exchange(h, xs != h->stream);
    if (s.bosonic) {
        exchange_front(h, xs);
        exchange_scalars(h, false, xs);
    }
    launch(h, PIMDB_K_BEAD_FORCES, [&] { launch_observable_terms(s, D, part, tiles, h->d_part, h->stream); },
           tile_launches(h));
    join_exchange(h, xs);
    std::vector<double> hp(n);
    double sc[4] = {0.0, 0.0, 0.0, 0.0};
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpyAsync(hp.data(), part, n * sizeof(double), cudaMemcpyDeviceToHost, h->stream);
    if (e == cudaSuccess && s.bosonic) e = cudaMemcpyAsync(sc, s.scal, sizeof sc, cudaMemcpyDeviceToHost, h->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(h->stream);
    if (e != cudaSuccess) return fail(h, PIMDB_ERR_CUDA, cudaGetErrorString(e));
    const int st = check_err_word(h);
    if (st != PIMDB_OK) return st;
    // assembled per bead as src/observables/{energy,classical,bosonic,
    // gsf_action}.cpp do on each bead's rank, then summed over beads
    // (observable.cpp:82-116)
    pimdb_observables o{};
    const double beta = 1.0 / (1.0 * h->cfg.temperature);
    for (int b = 0; b < P; ++b) {
        double t[7] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
        for (int q = 0; q < nb; ++q)
            for (int k = 0; k < 7; ++k) t[k] += hp[((size_t)b * nb + q) * 7 + k];
        const double spring = t[1] * (0.5 * s.kappa);
        double kinetic = 0.5 * D * N / beta;
        if (b == 0 && s.bosonic) kinetic += sc[1];
        else kinetic -= spring / P;
        o.kinetic += kinetic;
        o.potential += (t[2] + t[4]) / P;
        o.ext_pot += t[2] / P;
        o.int_pot += t[4] / P;
        o.virial += (t[3] + t[5]) * (0.5 / P);
        const double ke = t[0] * (0.5 / s.mass);
        o.temperature += 2.0 * ke / ((double)D * N * P * 1.0) / P / 3.1668152e-06;
        o.cl_kinetic += ke;
        o.cl_spring += (b == 0 && s.bosonic) ? sc[0] : spring;
        if (b == 0 && s.bosonic) {
            o.prob_dist += sc[2];
            o.prob_all += sc[3];
        }
        const double sp = s.kappa / P;
        const double pot_term = (t[2] + t[4]) / (3 * P);
        const double f2_term = t[6] / (9 * sp * P * P);
        o.w_gsf += ((b % 2 != 0) ? -pot_term : pot_term + f2_term) * (-beta);
        if (b % 2 != 0) o.pot_gsf += (t[2] + t[4]) / (0.5 * P);
    }
    if (h->d_nh) {
        // singleChainGetAdditionToH (nose_hoover.cpp:51-66) of every chain
        const NHPar& q = h->nh;
        const size_t m = (size_t)h->nh_chains * q.nchains;
        std::vector<double> eta(2 * m);
        CUDA_TRY(h, cudaMemcpy(eta.data(), h->d_nh, 2 * m * sizeof(double), cudaMemcpyDeviceToHost));
        const int ndof = q.variant == 0 ? D * N : (q.variant == 1 ? D : 1);
        for (long long ch = 0; ch < h->nh_chains; ++ch) {
            const double* et = &eta[(size_t)ch * q.nchains];
            const double* ed = &eta[m + (size_t)ch * q.nchains];
            double add = 0.5 * q.Q1 * ed[0] * ed[0];
            add += ndof * et[0] / q.thermo_beta;
            for (int i = 1; i < q.nchains; i++) {
                add += 0.5 * q.Qi * ed[i] * ed[i];
                add += et[i] / q.thermo_beta;
            }
            o.nh_energy += add;
        }
    }
    *out = o;
    return PIMDB_OK;
}

extern "C" int pimdb_local_energy(pimdb_handle* h, int n, const int* items, double* out) {
    if (!h || (n > 0 && (!items || !out)) || n < 0) return fail(h, PIMDB_ERR_ARG, "NULL argument or n < 0");
    if (n == 0) return PIMDB_OK;
    complete_pending(h);
    int* d_items = nullptr;
    double* d_out = nullptr;
    cudaError_t e = cudaMalloc((void**)&d_items, sizeof(int) * 2 * (size_t)n);
    if (e == cudaSuccess) e = cudaMalloc((void**)&d_out, sizeof(double) * (size_t)n);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(d_items, items, sizeof(int) * 2 * (size_t)n, cudaMemcpyHostToDevice, h->stream);
    if (e == cudaSuccess) {
        launch(h, PIMDB_K_BEAD_FORCES, [&] { launch_local_energy(h->s, h->D, n, d_items, d_out, h->stream); });
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(out, d_out, sizeof(double) * (size_t)n, cudaMemcpyDeviceToHost, h->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(h->stream);
    cudaFree(d_items);
    cudaFree(d_out);
    if (e != cudaSuccess) return fail(h, PIMDB_ERR_CUDA, cudaGetErrorString(e));
    return check_err_word(h);
}

extern "C" int pimdb_exchange_arrays(pimdb_handle* h, double* E_kn, double* V, double* Vb) {
    if (!h) return PIMDB_ERR_ARG;
    const Sys& s = h->s;
    if (!s.bosonic) return fail(h, PIMDB_ERR_CONFIG, "no exchange arrays for a distinguishable configuration");
    if (h->factorial) return fail(h, PIMDB_ERR_CONFIG, "the factorial exchange has no cycle energies or recursions");
    CUDA_TRY(h, cudaStreamSynchronize(h->stream));
    if (E_kn) CUDA_TRY(h, cudaMemcpy(E_kn, s.E, (size_t)s.N * (s.N + 1) / 2 * sizeof(double), cudaMemcpyDeviceToHost));
    if (V) CUDA_TRY(h, cudaMemcpy(V, s.V, (size_t)(s.N + 1) * sizeof(double), cudaMemcpyDeviceToHost));
    if (Vb) CUDA_TRY(h, cudaMemcpy(Vb, s.Vb, (size_t)(s.N + 1) * sizeof(double), cudaMemcpyDeviceToHost));
    return PIMDB_OK;
}

extern "C" int pimdb_profile(pimdb_handle* h, int enable, double* ms, long long* counts, long long* launches) {
    if (!h) return PIMDB_ERR_ARG;
    for (int k = 0; k < PIMDB_NUM_KERNEL_CLASSES; ++k) {
        if (ms) ms[k] = h->prof_ms[k];
        if (counts) counts[k] = h->prof_n[k];
    }
    if (launches) *launches = h->launches;
    if (enable >= 0) {
        CUDA_TRY(h, cudaStreamSynchronize(h->stream));
        h->profile = enable > 0;
        for (int k = 0; k < PIMDB_NUM_KERNEL_CLASSES; ++k) {
            h->prof_ms[k] = 0.0;
            h->prof_n[k] = 0;
        }
        h->launches = 0;
    }
    return PIMDB_OK;
}

// FP64 pipe throughput probe: independent fused multiply-add chains, no
// memory traffic.  Used as the measured FP64 peak of the roofline.
__global__ void k_fp64_fma_probe(double* out, int iters, double a, double b) {
    double r0 = threadIdx.x * 1e-9, r1 = r0 + 1e-9, r2 = r0 + 2e-9, r3 = r0 + 3e-9;
    double r4 = r0 + 4e-9, r5 = r0 + 5e-9, r6 = r0 + 6e-9, r7 = r0 + 7e-9;
    for (int i = 0; i < iters; ++i) {
        r0 = fma(r0, a, b); r1 = fma(r1, a, b); r2 = fma(r2, a, b); r3 = fma(r3, a, b);
        r4 = fma(r4, a, b); r5 = fma(r5, a, b); r6 = fma(r6, a, b); r7 = fma(r7, a, b);
    }
    const double s = r0 + r1 + r2 + r3 + r4 + r5 + r6 + r7;
    if (s == 1.2345) out[0] = s;  // keeps the chains alive
}

// FP32 pipe throughput probe: the same shape with float chains (the mixed
// paths' pair forces run on this pipe).
__global__ void k_fp32_fma_probe(float* out, int iters, float a, float b) {
    float r0 = threadIdx.x * 1e-6f, r1 = r0 + 1e-6f, r2 = r0 + 2e-6f, r3 = r0 + 3e-6f;
    float r4 = r0 + 4e-6f, r5 = r0 + 5e-6f, r6 = r0 + 6e-6f, r7 = r0 + 7e-6f;
    for (int i = 0; i < iters; ++i) {
        r0 = fmaf(r0, a, b); r1 = fmaf(r1, a, b); r2 = fmaf(r2, a, b); r3 = fmaf(r3, a, b);
        r4 = fmaf(r4, a, b); r5 = fmaf(r5, a, b); r6 = fmaf(r6, a, b); r7 = fmaf(r7, a, b);
    }
    const float s = r0 + r1 + r2 + r3 + r4 + r5 + r6 + r7;
    if (s == 1.2345f) out[0] = s;
}

extern "C" int pimdb_math_check(const double* x, int n, double* out) {
    if (!x || !out || n < 0) return PIMDB_ERR_ARG;
    if (n == 0) return PIMDB_OK;
    double* d = nullptr;
    CUDA_TRY(nullptr, cudaMalloc(&d, sizeof(double) * 9 * (size_t)n));
    cudaError_t e = cudaMemcpy(d, x, sizeof(double) * n, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) {
        launch_math_check(d, n, d + n, nullptr);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(out, d + n, sizeof(double) * 8 * (size_t)n, cudaMemcpyDeviceToHost);
    cudaFree(d);
    CUDA_TRY(nullptr, e);
    return PIMDB_OK;
}

extern "C" int pimdb_measure_fp64_peak(double* tflops) {
    if (!tflops) return PIMDB_ERR_ARG;
    int dev = 0, sms = 0;
    CUDA_TRY(nullptr, cudaGetDevice(&dev));
    CUDA_TRY(nullptr, cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    double* out = nullptr;
    CUDA_TRY(nullptr, cudaMalloc((void**)&out, sizeof(double)));
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    const int blocks = sms * 8, threads = 256, iters = 4096;
    k_fp64_fma_probe<<<blocks, threads>>>(out, iters, 0.999999, 1e-7);
    cudaEventRecord(e0);
    const int reps = 5;
    for (int r = 0; r < reps; ++r) k_fp64_fma_probe<<<blocks, threads>>>(out, iters, 0.999999, 1e-7);
    cudaEventRecord(e1);
    cudaEventSynchronize(e1);
    float ms = 0.f;
    cudaEventElapsedTime(&ms, e0, e1);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    cudaFree(out);
    CUDA_TRY(nullptr, cudaGetLastError());
    const double flops = 2.0 * 8.0 * iters * (double)threads * blocks * reps;
    *tflops = flops / (ms * 1e-3) / 1e12;
    return PIMDB_OK;
}

extern "C" int pimdb_measure_fp32_peak(double* tflops) {
    if (!tflops) return PIMDB_ERR_ARG;
    int dev = 0, sms = 0;
    CUDA_TRY(nullptr, cudaGetDevice(&dev));
    CUDA_TRY(nullptr, cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    float* out = nullptr;
    CUDA_TRY(nullptr, cudaMalloc((void**)&out, sizeof(float)));
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    const int blocks = sms * 8, threads = 256, iters = 65536;
    k_fp32_fma_probe<<<blocks, threads>>>(out, iters, 0.9999f, 1e-7f);
    cudaEventRecord(e0);
    const int reps = 5;
    for (int r = 0; r < reps; ++r) k_fp32_fma_probe<<<blocks, threads>>>(out, iters, 0.9999f, 1e-7f);
    cudaEventRecord(e1);
    cudaEventSynchronize(e1);
    float ms = 0.f;
    cudaEventElapsedTime(&ms, e0, e1);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    cudaFree(out);
    CUDA_TRY(nullptr, cudaGetLastError());
    const double flops = 2.0 * 8.0 * iters * (double)threads * blocks * reps;
    *tflops = flops / (ms * 1e-3) / 1e12;
    return PIMDB_OK;
}

extern "C" int pimdb_set_option(pimdb_handle* h, const char* name, int value) {
    if (!h || !name) return PIMDB_ERR_ARG;
    const std::string n(name);
    drop_graphs(h);
    if (n == "exact_exchange") h->opt_exact_exchange = value ? 1 : 0;
    else if (n == "fused_normal_modes") h->fused_nm = value && h->d_cmpart != nullptr;
    else if (n == "fft_normal_modes") {
        h->opt_fft = value ? 1 : 0;
        // the matrix transforms run in the block kernel only
        if (!value && h->fused_nm && !nm_block_fits(h->s, h->D)) h->fused_nm = false;
    }
    else if (n == "newton3") h->opt_newton3 = value ? 1 : 0;
    else if (n == "cell_lists") {
        if (value > 0 && !h->d_cells)
            return fail(h, PIMDB_ERR_CONFIG, "cell lists need a periodic box with at least 4 cutoff-wide cells per edge");
        h->opt_cells = value < 0 ? -1 : (value ? 1 : 0);
    } else if (n == "cuda_graphs") {
        h->opt_graph = value ? 1 : 0;
    } else if (n == "flat_energies") {
        h->s.eflat = value < 0 ? exchange_flat_default(h->s.N) : (value ? 1 : 0);
    } else if (n == "reserved_sms") {
        h->opt_reserved_sms = value < 0 ? -1 : value;
    } else if (n == "pair_entry_cap") {
        if (value < 0 || value > 1024 || value % 32)
            return fail(h, PIMDB_ERR_ARG, "pair_entry_cap must be 0 or a multiple of 32 up to 1024");
        h->s.pair_cap = value;
    } else return fail(h, PIMDB_ERR_ARG, "unknown option " + n);
    return PIMDB_OK;
}

// ---------------------------------------------------------------------------
// Fine-grained steps mirroring the reference's plugin calls one by one
// (Simulation::run, src/simulation.cpp:246-259).  They use the separate
// (unfused) kernels; pimdb_step composes the same operations.

extern "C" int pimdb_thermostat_step(pimdb_handle* h, int substep) {
    if (!h || substep < 0 || substep > 1) return PIMDB_ERR_ARG;
    const pimdb_config& c = h->cfg;
    complete_pending(h);  // finish the previous step's deferred work first
    if (substep == 0) draw_noise(h, h->step);  // the step's normals, as the reference draws them
    if (c.thermostat >= PIMDB_THERMO_NOSE_HOOVER) nose_hoover(h);
    else if (c.thermostat == PIMDB_THERMO_LANGEVIN && c.nmthermostat) nm_thermo(h, 0, substep);
    else if (c.thermostat == PIMDB_THERMO_LANGEVIN) cart(h, SF_LANGEVIN, substep, 0);
    CUDA_TRY(h, cudaGetLastError());
    return PIMDB_OK;
}

extern "C" int pimdb_zero_momentum(pimdb_handle* h) {
    if (!h) return PIMDB_ERR_ARG;
    complete_pending(h);
    cart(h, SF_COM_PARTIAL, 0, 0);
    cart(h, SF_COM_APPLY, 0, 0);
    CUDA_TRY(h, cudaGetLastError());
    return PIMDB_OK;
}

extern "C" int pimdb_propagate(pimdb_handle* h) {
    if (!h) return PIMDB_ERR_ARG;
    complete_pending(h);
    ++h->xgen;
    if (h->cfg.propagator == PIMDB_PROP_NORMAL_MODES) {
        h->modes_valid = false;
        launch(h, PIMDB_K_NM_PROPAGATE, [&] {
            launch_nm_propagate(h->s, h->D, h->d_C, h->d_T, h->d_rot, 0, h->d_red[0], 0,
                                h->opt_fft ? (const double2*)h->d_tw : nullptr, h->stream);
        });
        enqueue_forces(h);
        cart(h, SF_KICK, 0, 1);
    } else {
        cart(h, SF_KICK | SF_DRIFT, 0, 0);
        enqueue_forces(h);
        cart(h, SF_KICK, 0, 0);
    }
    CUDA_TRY(h, cudaGetLastError());
    return check_err_word(h);
}
