// Block- and warp-level pieces of the Feldman-Hirshberg exchange, shared by
// the one-system kernels (exchange.cu) and the batched-replica kernel
// (batch.cu).  Each function works on one system given by a Sys; the caller
// chooses which block or warp runs it.
#pragma once

#include <math_constants.h>

#include "common.cuh"
#include "forces_dev.cuh"  // exp_tang
#include "kernels.h"       // the exchange's flag indices

namespace pimdb {
__device__ __forceinline__ size_t tri(int v) { return (size_t)v * (size_t)(v + 1) / 2; }

template <int D>
__device__ __forceinline__ double sepsq(const Sys& s, int ba, int ia, int bb, int ib) {
    // |x_bb[ib] - x_ba[ia]|^2 with the minimum image (bosonic_exchange_base.cpp:30-64)
    double d2 = 0.0;
#pragma unroll
    for (int a = 0; a < D; ++a) {
        double d = s.x[idx<D>(s, bb, a, ib)] - s.x[idx<D>(s, ba, a, ia)];
        if (s.pbc) d = min_image(d, s.L, s.invL);
        d2 += d * d;
    }
    return d2;
}
// One warp per row v: E[v][v] = k/2 |xP_v - x1_v|^2, then
// E[v][u] = E[v][u+1] + k/2 (|x1_{u+1} - xP_u|^2 - |xP_v - x1_{u+1}|^2 + |xP_v - x1_u|^2)
// for u = v-1 .. 0, evaluated as a warp-wide suffix scan over u.  The middle
// distance of entry u is the last distance of entry u+1, so each entry costs
// two distance evaluations (passed between lanes by a shuffle), or one with
// `link` (link[u] = |x1_{u+1} - xP_u|^2, computed once per u by the caller).
template <int D>
__device__ inline void energy_row(const Sys& s, int v, int lane, const double* link = nullptr) {
    const int first = 0, last = s.P - 1;
    const double hk = 0.5 * s.kappa;
    double* row = s.E + tri(v);
    double xv[D];
#pragma unroll
    for (int a = 0; a < D; ++a) xv[a] = s.x[idx<D>(s, last, a, v)];
    auto dist_to_v = [&](int u) {  // |xP_v - x1_u|^2
        double d2 = 0.0;
#pragma unroll
        for (int a = 0; a < D; ++a) {
            double d = xv[a] - s.x[idx<D>(s, first, a, u)];
            if (s.pbc) d = min_image(d, s.L, s.invL);
            d2 += d * d;
        }
        return d2;
    };
    double cnext = dist_to_v(v);  // |xP_v - x1_{u+1}|^2 for the lane holding u = base
    double carry = hk * cnext;
    if (lane == 0) row[v] = carry;
    for (int base = v - 1; base >= 0; base -= 32) {
        const int u = base - lane;
        const double c = u >= 0 ? dist_to_v(u) : 0.0;
        double cu1 = __shfl_up_sync(0xffffffffu, c, 1);
        if (lane == 0) cu1 = cnext;
        double term = 0.0;
        if (u >= 0) term = hk * ((link ? link[u] : sepsq<D>(s, last, u, first, u + 1)) - cu1 + c);
        cnext = __shfl_sync(0xffffffffu, c, 31);
        // inclusive scan over lanes (lane 0 holds the largest u)
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const double y = __shfl_up_sync(0xffffffffu, term, o);
            if (lane >= o) term += y;
        }
        if (u >= 0) {
            const double e = carry + term;
            row[u] = e;
            // backward node r = N - u depends on node r' = N - 1 - v
            if (u >= 1) s.Et[tri(s.N - u - 1) + (s.N - 1 - v)] = e;
        }
        carry += __shfl_sync(0xffffffffu, term, 31);
    }
    if (lane == 0 && v >= 1) s.Et[tri(s.N - v - 1) + (s.N - 1 - v)] = row[v];
}
// The recursions as "node" recursions.  Forward: node n = level m = n,
// node 0 known (V = 0), node n depends on nodes u < n through the packed row
// E[n-1][u].  Backward: node r = N - l, node 0 (l = N) known, node r depends
// on nodes r' < r through Et[r-1][r'] = E[p][l] with p = N - 1 - r' (so
// p + 1 = N - r').  Both are evaluated by the same blocked scheme: nodes are
// taken 32 at a time; one warp resolves the 32 nodes of a block one after the
// other with shuffles (no barrier), and the finished block is folded into the
// accumulators of all later nodes.
constexpr int kWaveThreads = 256;

// ---- FP32 estimate.  In base-2 logarithms, with b = beta log2(e): node n's
// log-sum is L_n = log2 sum_{u<n} 2^(g_u - b E[n-1][u]), and what it
// contributes to later nodes is g_n = L_n - log2(n) forward (g_0 = 0),
// g_n = L_n - log2(N - n) backward (g_0 = -log2(N)).  Forward V_n = -g_n / b,
// backward value -L_n / b.  A running log-sum is a pair (mx, sm): 2^mx sm.
__device__ __forceinline__ float ex2f(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float lg2f(float x) {
    float y;
    asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// E for the estimate, from the double's upper word alone: sign, exponent and
// 20 fraction bits (2^-20 relative is far below what the estimate needs; half
// the bytes, no FP64-pipe conversion), 0 and 2^127 beyond a float's range.
// est_load is volatile so that a thread's loads are all issued where they
// stand instead of one by one in front of their uses (one L2 round trip per
// block of nodes, not 32).
__device__ __forceinline__ unsigned est_load(const double* p) {
    unsigned v;
    asm volatile("ld.global.cg.u32 %0, [%1];" : "=r"(v) : "l"(reinterpret_cast<const unsigned*>(p) + 1));
    return v;
}
__device__ __forceinline__ float est_value(unsigned hi) {
    const unsigned e = (hi >> 20) & 0x7ffu;
    if (e < 1023u - 126u) return 0.0f;
    const unsigned q = e > 1023u + 126u ? 254u << 23 : (e - 896u) << 23 | (hi & 0xfffffu) << 3;
    return __uint_as_float(hi & 0x80000000u | q);
}
struct EstDir {
    const double* E;  // packed rows (s.E forward, s.Et backward)
    int nn, N;
    float b;  // beta log2(e)
    bool fwd;
    __device__ EstDir(const Sys& s, int dir)
        : E(dir == 0 ? s.E : s.Et), nn(dir == 0 ? s.N + 1 : s.N), N(s.N),
          b((float)(s.beta_ex * 1.4426950408889634)), fwd(dir == 0) {}
    __device__ float norm(int n) const { return lg2f((float)(fwd ? n : N - n)); }
};
// One warp resolves the 32 nodes base .. base + 31: the lane's node's log-sum
// over earlier blocks in (mx, sm), its row's entries of this block in e.
// Returns g of the lane's node.
__device__ __forceinline__ float est_diagonal(const EstDir& d, int base, int lane, float mx, float sm,
                                              const unsigned (&e)[32]) {
    const int n = base + lane;
    const float nl = n >= 1 && n < d.nn ? d.norm(n) : 0.0f;
    float g = 0.0f;
#pragma unroll
    for (int t = 0; t < 32; ++t) {
        if (lane == t) g = n == 0 ? (d.fwd ? 0.0f : -d.norm(0)) : mx + lg2f(sm) - nl;
        const float gt = __shfl_sync(0xffffffffu, g, t);
        const float x = fmaf(-d.b, est_value(e[t]), gt), m = fmaxf(mx, x);
        const float z = fmaf(sm, ex2f(mx - m), ex2f(x - m));
        if (lane > t) {
            sm = z;
            mx = m;
        }
    }
    return g;
}
// The lane's row entries of the diagonal block (0 where there are none).
__device__ __forceinline__ void est_load_diagonal(const EstDir& d, int base, int lane, unsigned (&e)[32]) {
    const int n = base + lane;
    const bool row = n < d.nn && n >= 1;
    const double* at = d.E + (row ? tri(n - 1) + base : 0);
#pragma unroll
    for (int t = 0; t < 32; ++t) {
        e[t] = 0u;
        if (row && t < lane) e[t] = est_load(at + t);
    }
}
// Entries of row m against the 32 nodes of block j, four per thread of the
// row's eight (columns part, part + 8, ...).
__device__ __forceinline__ void est_load_row(const EstDir& d, int m, int j, int part, unsigned (&e)[4]) {
    const double* row = d.E + tri(m - 1) + 32 * j + part;
#pragma unroll
    for (int q = 0; q < 4; ++q) e[q] = est_load(row + 8 * q);
}
// Folds block j's nodes (gj[0..31]) into row m's log-sum; the eight threads
// of a row call it together (`valid` false: only to take part).
__device__ __forceinline__ void est_fold(const EstDir& d, const unsigned (&e)[4], const float* gj, int part, bool valid,
                                         float* mx, float* sm) {
    float t[4], m = -CUDART_INF_F;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        t[q] = fmaf(-d.b, est_value(e[q]), gj[part + 8 * q]);
        m = fmaxf(m, t[q]);
    }
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    float z = 0.0f;
#pragma unroll
    for (int q = 0; q < 4; ++q) z += ex2f(t[q] - m);
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) z += __shfl_xor_sync(0xffffffffu, z, o);
    if (part == 0 && valid) {
        const float a = *mx, n = fmaxf(a, m);
        *sm = fmaf(*sm, ex2f(a - n), z * ex2f(m - n));
        *mx = n;
    }
}
// The estimate of node n into s.Vh / s.Vbh.
__device__ __forceinline__ void est_store(const Sys& s, const EstDir& d, int n, float g) {
    if (d.fwd) s.Vh[n] = (double)(-g / d.b);
    else s.Vbh[d.N - n] = (double)(n == 0 ? 0.0f : -(g + d.norm(n)) / d.b);
    if (!d.fwd && n == 0) s.Vbh[0] = 0.0;
}

// Pass 1 of one direction (0 forward, 1 backward) by `nt` threads (whole
// warps, thread `t` of them; barrier `bar`, 0 for a whole block); `fsm` holds 3 (N + 1) floats.
// Warp 0 resolves block b + 1 while the other warps fold block b into the
// rows after it.  Both directions of N = 256 by one block of 256 threads, half
// each: 72 us (one after the other with one thread per row, loads one by one:
// about 300 us).  Out of line: a rare path whose arrays would otherwise set
// the callers' registers.
static __device__ __noinline__ void estimate_group(const Sys& s, int dir, float* fsm, int t, int nt, int bar) {
    const EstDir d(s, dir);
    const int nn = d.nn, lane = t & 31, warp = t >> 5;
    float* g = fsm;
    float* mx = fsm + (s.N + 1);
    float* sm = fsm + 2 * (s.N + 1);
    // barriers by constant ids: a block is charged for the ids it may use
    auto sync = [&] {
        if (bar == 0) __syncthreads();
        else if (bar == 1) asm volatile("bar.sync 1, %0;" ::"r"(nt) : "memory");
        else asm volatile("bar.sync 2, %0;" ::"r"(nt) : "memory");
    };
    for (int n = t; n < nn; n += nt) {
        mx[n] = -CUDART_INF_F;
        sm[n] = 0.0f;
    }
    sync();
    // warp 0: the diagonal block's entries loaded ahead of their turn
    unsigned e[32];
    auto diagonal = [&](int b) {
        const int n = 32 * b + lane;
        const float v = est_diagonal(d, 32 * b, lane, n < nn ? mx[n] : 0.0f, n < nn ? sm[n] : 1.0f, e);
        if (n < nn) {
            g[n] = v;
            est_store(s, d, n, v);
        }
    };
    // rows lo .. hi - 1 against block j, by the threads t0 .. nt - 1; each
    // warp takes eight rows at a time, every load issued before the first fold
    auto fold = [&](int lo, int hi, int j, int t0) {
        const int part = t & 7;
        for (int m0 = lo + ((t - t0) >> 5) * 8 + (lane >> 3); m0 - (lane >> 3) < hi; m0 += ((nt - t0) >> 5) * 8) {
            unsigned ea[4] = {0u, 0u, 0u, 0u}, eb[4] = {0u, 0u, 0u, 0u};
            const bool va = m0 < hi, vb = m0 + 4 < hi;
            if (va) est_load_row(d, m0, j, part, ea);
            if (vb) est_load_row(d, m0 + 4, j, part, eb);
            est_fold(d, ea, g + 32 * j, part, va, mx + m0, sm + m0);
            est_fold(d, eb, g + 32 * j, part, vb, mx + m0 + 4, sm + m0 + 4);
        }
    };
    const int nb = (nn + 31) / 32;
    if (warp == 0) {
        est_load_diagonal(d, 0, lane, e);
        diagonal(0);
    }
    sync();
    for (int b = 0; b + 1 < nb; ++b) {
        const int next = 32 * (b + 1), after = min(nn, next + 32);
        if (warp == 0) est_load_diagonal(d, next, lane, e);
        fold(next, after, b, 0);
        sync();
        if (warp == 0) diagonal(b + 1);
        if (nt == 32) fold(after, nn, b, 0);
        else if (warp > 0) fold(after, nn, b, 32);
        sync();
    }
}
// One direction by the whole block; `fsm` holds 3 (N + 1) floats.
__device__ inline void estimate_direction(const Sys& s, int dir, float* fsm) {
    estimate_group(s, dir, fsm, threadIdx.x, blockDim.x, 0);
}
// Both directions by the whole block, side by side on half its warps each;
// `fsm` holds 6 (N + 1) floats.
__device__ inline void estimate_both(const Sys& s, float* fsm) {
    const int nw = blockDim.x >> 5, h = nw / 2 * 32;
    if (nw < 2) {
        estimate_direction(s, 0, fsm);
        estimate_direction(s, 1, fsm);
    } else if ((int)threadIdx.x < h) {
        estimate_group(s, 0, fsm, threadIdx.x, h, 1);
    } else {
        estimate_group(s, 1, fsm + 3 * (s.N + 1), threadIdx.x - h, blockDim.x - h, 2);
    }
}

// FP64 triangular node solve: y(0) = 1, y(n) = sum_{u<n} W[n-1][u] y(u).
__device__ inline void blocked_solve(const double* __restrict__ W, int nn, double* y, double* acc) {
    const int tid = threadIdx.x, bd = blockDim.x, lane = tid & 31, warp = tid >> 5;
    for (int n = tid; n < nn; n += bd) acc[n] = 0.0;
    __syncthreads();
    const int nb = (nn + 31) / 32;
    for (int b = 0; b < nb; ++b) {
        const int base = 32 * b;
        if (warp == 0) {
            const int n = base + lane;
            double a = n == 0 ? 1.0 : (n < nn ? acc[n] : 0.0);
            double w[32];
#pragma unroll
            for (int t = 0; t < 32; ++t) w[t] = (n < nn && n >= 1 && t < lane) ? W[tri(n - 1) + base + t] : 0.0;
#pragma unroll
            for (int t = 0; t < 32; ++t) {
                const double yt = __shfl_sync(0xffffffffu, a, t);
                if (lane > t) a = fma(w[t], yt, a);
            }
            if (n < nn) y[n] = a;
        }
        __syncthreads();
        for (int m = base + 32 + tid; m < nn; m += bd) {
            const double* row = W + tri(m - 1) + base;
            double sacc = acc[m];
#pragma unroll 8
            for (int q = 0; q < 32; ++q) sacc = fma(row[q], y[base + q], sacc);
            acc[m] = sacc;
        }
        __syncthreads();
    }
}
// Pass 2: the FP64 weights of packed entry (row p, column u), both directions
// (dir 0 forward only, 1 backward only, -1 both); `inv` = 1/(p+1), once per
// row.  `tbl`: the exp_tang table (32 entries: a weights block then still
// fits beside the pair kernel's resident blocks) in shared memory (null:
// CUDA's exp).  Arguments of 709 and more give infinity either way (the
// solve then retries).
// 1/(p+1) for p < 4096, evaluated by the compiler (IEEE division, the
// device's own result) into constant memory: the weights read it once per row
// (a uniform index, one broadcast) instead of dividing.
struct RecipTable {
    double v[4096];
    constexpr RecipTable() : v() {
        for (int i = 0; i < 4096; ++i) v[i] = 1.0 / (i + 1);
    }
};
static __constant__ RecipTable kRecip = RecipTable();
__device__ __forceinline__ double recip_row(int p) { return p < 4096 ? kRecip.v[p] : 1.0 / (p + 1); }

__device__ __forceinline__ double weight_exp(double x, const double* tbl) {
    if (!tbl) return exp(x);
    return x < 709.0 ? exp_tang(x, tbl) : (double)INFINITY;
}
// Returns whether either weight it wrote is nonzero (the solve's band: node
// p + 1 depends on node u, backward node N - u on node N - 1 - p, both at
// distance p + 1 - u).
__device__ __forceinline__ bool exch_weight(const Sys& s, int p, int u, double inv, const double* tbl = nullptr,
                                            int dir = -1) {
    const double beta = s.beta_ex;
    const size_t e = tri(p) + u;
    const double E = s.E[e];
    bool nz = false;
    if (dir <= 0) {
        const double w = weight_exp(-beta * (E + s.Vh[u] - s.Vh[p + 1]), tbl) * inv;
        s.Wf[e] = w;
        nz = w != 0.0;
    }
    // backward node r = N - u from node r' = N - 1 - p (u >= 1)
    if (dir != 0 && u >= 1) {
        const double w = weight_exp(-beta * (E + s.Vbh[p + 1] - s.Vbh[u]), tbl) * inv;
        s.Wb[tri(s.N - u - 1) + (s.N - 1 - p)] = w;
        nz = nz || w != 0.0;
    }
    return nz;
}
// One direction's weights by the whole block (the in-block retry).
__device__ inline void weights_direction(const Sys& s, int dir, const double* tbl) {
    for (int p = 0; p < s.N; ++p) {
        const double inv = recip_row(p);
        for (int u = threadIdx.x; u <= p; u += blockDim.x) exch_weight(s, p, u, inv, tbl, dir);
    }
}
// The weights of every packed entry (row p, column u), both directions, as
// exch_weight computes them, in double-float on the FP32 pipe, by one block
// (the batched engine's mixed path; the one block that ran a fresh
// estimate): w = exp(-beta (E + Vh_u - Vh_{p+1})) / (p + 1) forward,
// exp(-beta (E + Vbh_{p+1} - Vbh_u)) / (p + 1) backward.  Arguments above 88 give infinity (the solve then retries with a
// fresh estimate or the exact recursion), below -88 zero (a weight under
// 1e-38 of the ones that normalise the row).  `vsm` holds 4 (N + 1) floats.
// Returns this thread's band: the largest p + 1 - u of a nonzero weight.
// weights_df_block_f64arg forms the argument in FP64 (only the exponential
// in double-float): E, Vh_u and Vh_{p+1} are up to beta_ex V_B ~ 10^3-10^4 kT
// and nearly cancel, so 48 bits of each leave 1e-11 in the weight.  Entries
// whose FP32 argument is below -89 by more than its own roundings (below 3e-7
// of its terms) are zero without any FP64 operation.
// That an entry at -89 does not count takes a row whose largest is near 0: an
// estimate that follows the energies to a few kT.  It is formed from 20 bits
// of them, so potentials above kWideKT may be off by more (rings stretched far
// beyond equilibrium): weights_wide then.
constexpr double kWideKT = 4194304.0;  // 2^22: 2^-20 of it, a few times, is about 16 kT
// The weights with CUDA's exp over its whole range (out of line: a rare path).
static __device__ __noinline__ int weights_wide(const Sys& s) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int N = s.N;
    const double nbeta = -s.beta_ex;
    int band = 0;
    for (int p = warp; p < N; p += nw) {
        const double inv = recip_row(p), vp = s.Vh[p + 1], vbp = s.Vbh[p + 1];
        for (int u = lane; u <= p; u += 32) {
            const double E = __ldcg(s.E + tri(p) + u);
            const double wf = exp(nbeta * (E + s.Vh[u] - vp)) * inv;
            const double wb = u >= 1 ? exp(nbeta * (E + vbp - s.Vbh[u])) * inv : 0.0;
            s.Wf[tri(p) + u] = wf;
            if (u >= 1) s.Wb[tri(N - u - 1) + (N - 1 - p)] = wb;
            if (wf != 0.0 || wb != 0.0) band = max(band, p + 1 - u);
        }
    }
    return band;
}
__device__ inline int weights_df_block_f64arg(const Sys& s, const dfl::ExpTable& etbl, float* vsm) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int N = s.N;
    double* vh = reinterpret_cast<double*>(vsm);
    double* vbh = vh + N + 1;
    const double nbeta = -s.beta_ex;
    const float nbf = round_f32(nbeta);
    int wide = 0;
    for (int m = threadIdx.x; m <= N; m += blockDim.x) {
        vh[m] = s.Vh[m];
        vbh[m] = s.Vbh[m];
        if (!(fabs(nbeta * vh[m]) <= kWideKT && fabs(nbeta * vbh[m]) <= kWideKT)) wide = 1;
    }
    if (__syncthreads_or(wide)) return weights_wide(s);
    int band = 0;
    for (int p = warp; p < N; p += nw) {
        const dfl::df inv = split_df(recip_row(p));
        const double vp = vh[p + 1], vbp = vbh[p + 1];
        const float vpf = round_f32(vp), vbpf = round_f32(vbp);
        const size_t r = tri(p);
        auto weight = [&](double E, double a, double b, float Ef, float af, float bf) {
            const float quick = Ef + (af - bf) - 4e-7f * (fabsf(Ef) + fabsf(af) + fabsf(bf));
            if (nbf * quick < -89.0f) return 0.0;
            const double x = nbeta * (E + a - b);
            return df_to_f64(dfl::mul(dfl::exp(split_df(x), etbl), inv));
        };
        // four 32-entry chunks at a time, their loads issued together (the
        // rows were just written by other SMs: an L2 round trip per group)
        for (int u0 = lane; u0 <= p; u0 += 128) {
            double E[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) E[k] = u0 + 32 * k <= p ? __ldcg(s.E + r + u0 + 32 * k) : 0.0;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int u = u0 + 32 * k;
                if (u > p) break;
                const double vu = vh[u];
                const float Ef = round_f32(E[k]);
                const double wf = weight(E[k], vu, vp, Ef, round_f32(vu), vpf);
                s.Wf[r + u] = wf;
                bool nz = !f64_is_zero(wf);
                if (u >= 1) {
                    const double vbu = vbh[u];
                    const double wb = weight(E[k], vbp, vbu, Ef, vbpf, round_f32(vbu));
                    s.Wb[tri(N - u - 1) + (N - 1 - p)] = wb;
                    nz = nz || !f64_is_zero(wb);
                }
                if (nz) band = max(band, p + 1 - u);
            }
        }
    }
    return band;
}
// Rows warp, warp + nw, ...
__device__ inline int weights_df_block(const Sys& s, const dfl::ExpTable& etbl, float* vsm, int warp, int nw) {
    using dfl::df;
    const int lane = threadIdx.x & 31;
    const int N = s.N;
    float* vh = vsm;               // Vh hi, lo
    float* vbh = vsm + 2 * (N + 1);  // Vbh hi, lo
    for (int m = threadIdx.x; m <= N; m += blockDim.x) {
        split_f32(s.Vh[m], vh[m], vh[N + 1 + m]);
        split_f32(s.Vbh[m], vbh[m], vbh[N + 1 + m]);
    }
    __syncthreads();
    const df nbeta = dfl::neg(split_df(s.beta_ex));
    int band = 0;
    for (int p = warp; p < N; p += nw) {
        const df inv = split_df(recip_row(p));
        const df vp = dfl::fast_two_sum(vh[p + 1], vh[N + 2 + p]);
        const df vbp = dfl::fast_two_sum(vbh[p + 1], vbh[N + 2 + p]);
        const size_t r = tri(p);
        for (int u = lane; u <= p; u += 32) {
            const df E = split_df(s.E[r + u]);
            const df vu = dfl::fast_two_sum(vh[u], vh[N + 1 + u]);
            const df tf = dfl::add(dfl::add(E, vu), dfl::neg(vp));
            const double wf = df_to_f64(dfl::mul(dfl::exp(dfl::mul(nbeta, tf), etbl), inv));
            s.Wf[r + u] = wf;
            bool nz = !f64_is_zero(wf);
            if (u >= 1) {
                const df vbu = dfl::fast_two_sum(vbh[u], vbh[N + 1 + u]);
                const df tb = dfl::add(dfl::add(E, vbp), dfl::neg(vbu));
                const double wb = df_to_f64(dfl::mul(dfl::exp(dfl::mul(nbeta, tb), etbl), inv));
                s.Wb[tri(N - u - 1) + (N - 1 - p)] = wb;
                nz = nz || !f64_is_zero(wb);
            }
            if (nz) band = max(band, p + 1 - u);
        }
    }
    return band;
}

// Exact level-by-level FP64 log-sum-exp in the reference's order (used only
// when the estimate is unusable, or on request).  `vs` holds N+1 doubles,
// `red` 32.
__device__ inline void exact_forward(const Sys& s, double* vs, double* red) {
    const int N = s.N, tid = threadIdx.x, bd = blockDim.x;
    const double beta = s.beta_ex;
    if (tid == 0) vs[0] = 0.0;
    __syncthreads();
    for (int m = 1; m <= N; ++m) {
        const double* row = s.E + tri(m - 1);
        double lmin = 1.79769313486231570815e308;
        for (int u = tid; u < m; u += bd) lmin = fmin(lmin, row[u] + vs[u]);
        const double shift = block_min(lmin, red);
        double ls = 0.0;
        for (int u = tid; u < m; u += bd) ls += exp(-beta * (row[u] + vs[u] - shift));
        const double tot = block_sum(ls, red);
        if (tid == 0) vs[m] = shift - (1.0 / beta) * log(tot / (double)m);
        __syncthreads();
    }
}
__device__ inline void exact_backward(const Sys& s, double* vs, double* red) {
    const int N = s.N, tid = threadIdx.x, bd = blockDim.x;
    const double beta = s.beta_ex;
    if (tid == 0) vs[N] = 0.0;
    __syncthreads();
    for (int l = N - 1; l > 0; --l) {
        double lmin = 1.79769313486231570815e308;
        for (int p = l + tid; p < N; p += bd) lmin = fmin(lmin, s.E[tri(p) + l] + vs[p + 1]);
        const double shift = block_min(lmin, red);
        double ls = 0.0;
        for (int p = l + tid; p < N; p += bd) ls += exp(-beta * (s.E[tri(p) + l] + vs[p + 1] - shift)) / (p + 1);
        const double tot = block_sum(ls, red);
        if (tid == 0) vs[l] = shift - log(tot) / beta;
        __syncthreads();
    }
}
// |log y| above which the next evaluation computes a fresh FP32 estimate
// instead of reusing the current potentials, and above which the present
// evaluation switches to the exact level-by-level recursion.
constexpr int kGridSolveMinN = 768;     // from here the solve runs across SMs
constexpr int kFlatEnergiesMinN = 512;  // from here the cycle energies come from link prefix sums
constexpr int kGridSolveCtas = 64;      // CTAs per direction
constexpr int kGridSolveThreads = 256;
constexpr double kRefreshLogY = 30.0;
constexpr double kExactLogY = 200.0;
// Pass 3, one direction (0 forward, 1 backward) by the whole block: the y
// solve and the exact V / V_backwards.  `ys` holds 2 (N+1) + 32 doubles.
// When the solve is unusable (|log y| >= 200) and `allow_exact` is 0 (the
// estimate was the previous evaluation's potentials, not a fresh FP32
// recursion), no exact recursion is run: xflags[6] asks the caller to
// retry with a fresh estimate instead.
// `pre`: y of this direction already solved (k_exch_solve_grid), or null.
// Returns 1 when it gave up that way (block-uniform); with `flag_retry` 0
// xflags[6] is left alone (the caller retries in the same block).
// `et` (2^(j/256) as double-floats in shared memory): log y in double-float
// on the FP32 pipe (log_df); null: CUDA's FP64 log.
__device__ inline int solve_direction(const Sys& s, int dir, int force_exact, double* ys, int allow_exact = 1,
                                      const double* pre = nullptr, int flag_retry = 1,
                                      const dfl::ExpTable* et = nullptr) {
    double* acc = ys + s.N + 1;
    double* red = ys + 2 * (s.N + 1);
    const int N = s.N, tid = threadIdx.x, bd = blockDim.x;
    int bad = force_exact, stale = 0;
    if (dir == 0) {
        if (!force_exact) {
            if (pre) {
                for (int m = tid; m <= N; m += bd) ys[m] = ((volatile const double*)pre)[m];
                __syncthreads();
            } else {
                blocked_solve(s.Wf, N + 1, ys, acc);
            }
            for (int m = tid; m <= N; m += bd) {
                const double y = ys[m];
                const double ly = et ? log_df(y, *et) : log(y);
                if (!(y > 0.0) || !(fabs(ly) < kExactLogY)) bad = 1;
                if (!(fabs(ly) < kRefreshLogY)) stale = 1;
                s.yf[m] = y;
                s.V[m] = s.Vh[m] - ly * s.inv_beta_ex;
            }
        }
        bad = __syncthreads_or(bad);
        if (bad && !allow_exact) {
            if (tid == 0 && flag_retry) s.xflags[6] = 1;
            return 1;
        }
        if (bad) {
            exact_forward(s, ys, red);
            for (int m = tid; m <= N; m += bd) s.V[m] = ys[m];
        }
        int nonfinite = 0;
        __syncthreads();
        for (int m = tid; m <= N; m += bd)
            if (!isfinite(s.V[m])) nonfinite = 1;
        nonfinite = __syncthreads_or(nonfinite);
        stale = __syncthreads_or(stale);
        if (tid == 0) {
            s.xflags[0] = bad;
            s.xflags[4] = (stale ? 1 : 0) | (nonfinite ? 2 : 0);
            if (nonfinite) atomicOr(s.err, ERRB_NONFINITE_VB);
        }
    } else {
        if (!force_exact) {
            // nodes r = 0..N-1 <-> levels l = N..1
            if (pre) {
                for (int r = tid; r < N; r += bd) ys[r] = ((volatile const double*)pre)[r];
                __syncthreads();
            } else {
                blocked_solve(s.Wb, N, ys, acc);
            }
            for (int l = tid + 1; l < N; l += bd) {
                const double y = ys[N - l];
                const double ly = et ? log_df(y, *et) : log(y);
                if (!(y > 0.0) || !(fabs(ly) < kExactLogY)) bad = 1;
                if (!(fabs(ly) < kRefreshLogY)) stale = 1;
                s.yb[l] = y;
                s.Vb[l] = s.Vbh[l] - ly * s.inv_beta_ex;
            }
        }
        if (tid == 0) {
            s.Vb[N] = 0.0;
            s.yb[N] = 1.0;
        }
        bad = __syncthreads_or(bad);
        if (bad && !allow_exact) {
            if (tid == 0 && flag_retry) s.xflags[6] = 1;
            return 1;
        }
        if (bad) {
            exact_backward(s, ys, red);
            for (int l = tid + 1; l <= N; l += bd) s.Vb[l] = ys[l];
        }
        int nonfinite = 0;
        __syncthreads();
        for (int l = tid + 1; l <= N; l += bd)
            if (!isfinite(s.Vb[l])) nonfinite = 1;
        nonfinite = __syncthreads_or(nonfinite);
        stale = __syncthreads_or(stale);
        if (tid == 0) {
            s.xflags[1] = bad;
            s.xflags[5] = (stale ? 1 : 0) | (nonfinite ? 2 : 0);
            if (nonfinite) atomicOr(s.err, ERRB_NONFINITE_VB);
        }
    }
    return 0;
}
// After both directions (one block): the per-row factors of the connection
// probabilities, which need both V and V_backwards, and the estimates of the
// next evaluation: V, V_backwards themselves or, with `extrapolate` and a
// previous result in s.Vp (NaN until there is one), the linear extrapolation
// 2 V(t) - V(t - dt), which smooth dynamics keep much closer.  The caller
// asks for no extrapolation after an evaluation from a fresh estimate: the
// coordinates may have jumped, and 2 V - V(before the jump) would fail again
// (one more fresh estimate, 0.63 ms at N = 4096).  An estimate that was not
// extrapolated and is 30 kT off asks for no fresh one either: the next, which
// is, will be far closer.  With `et` the row exponentials in double-float
// (exp_df).
__device__ inline void solve_finish(const Sys& s, int extrapolate = 0, const dfl::ExpTable* et = nullptr) {
    const int N = s.N, tid = threadIdx.x, bd = blockDim.x;
    const double beta = s.beta_ex;
    volatile double* V = s.V;
    volatile double* Vb = s.Vb;
    const double VN = V[N];
    for (int l = tid; l < N; l += bd) {
        const double vbl = Vb[l + 1];
        const double aR = -beta * (s.Vh[l + 1] + vbl - VN), aC = -beta * (V[l + 1] + vbl - VN);
        s.rowR[l] = et ? exp_df(aR, *et) : exp(aR);
        s.rowC[l] = et ? exp_df(aC, *et) : exp(aC);
    }
    __syncthreads();
    // [4], [5] per direction: 1 the estimate was 30 kT off, 2 not finite
    const int off = ((volatile int*)s.xflags)[4] | ((volatile int*)s.xflags)[5];
    const int need = (off & 2) || ((off & 1) && (!s.Vp || ((volatile int*)s.xflags)[kExchOrder]));
    for (int m = tid; m <= N; m += bd) {
        const double v = V[m], vb = m >= 1 ? Vb[m] : 0.0;
        if (s.Vp && extrapolate && isfinite(s.Vp[m]) && isfinite(s.Vp[N + 1 + m])) {
            s.Vh[m] = 2.0 * v - s.Vp[m];
            s.Vbh[m] = 2.0 * vb - s.Vp[N + 1 + m];
        } else {
            s.Vh[m] = v;
            s.Vbh[m] = vb;
        }
        if (s.Vp) {
            s.Vp[m] = v;
            s.Vp[N + 1 + m] = vb;
        }
    }
    __syncthreads();  // every thread has read the flags
    if (tid == 0) {
        s.xflags[2] = 0;
        s.xflags[3] = need;
        if (s.Vp) s.xflags[kExchOrder] = extrapolate;
        s.Vb[0] = VN;  // V_backwards[0] = V[N] (:127)
        s.scal[0] = VN;
    }
}
// Exterior spring forces (:159-215).  Warps [0, N) handle bead P (row l of
// the connection-probability matrix), warps [N, 2N) bead 1 (column l).
// Probabilities: close-cycle P[l][u] = Wf[l][u] y_u R_l (u <= l), direct
// link P[l][l+1] = 1 - C_l; with the exact fallback they are evaluated
// from their defining exponentials.  When `accumulate`, the spring force is
// added to f (which holds the physical forces; simulation.cpp:363-373).
// `xs` (optional): the positions of beads 1 and P staged in shared memory,
// xs[(side * D + a) * N + i] with side 0 = bead 1, 1 = bead P.
template <int D>
// With `adjoint` set, the row writes the cotangent of the exchange potential
// instead of the force: fx = vb_bar * dV_B/dx = -vb_bar * kappa * sum, with
// neither the interior neighbour spring nor the accumulation into f.
// `band` > 0: every weight beyond that distance from the diagonal is exactly
// zero (the banded solve's measurement); the rows skip the 32-entry chunks
// that hold only such entries, each lane keeping its own entries (the same
// sums, bit for bit).
__device__ inline void exch_force_row(const Sys& s, int w, int lane, int accumulate, const double* xs = nullptr,
                                      int adjoint = 0, double vb_bar = 0.0, int band = 0) {
    const int N = s.N;
    const double beta = s.beta_ex;
    const double VN = s.V[N];
    const bool exact = s.xflags[0] != 0;
    const int first = 0, last = s.P - 1;
    double sum[D];
#pragma unroll
    for (int a = 0; a < D; ++a) sum[a] = 0.0;
    int bead, nb, l;
    if (w < N) {  // last bead, particle l: sum over n <= l+1
        l = w;
        bead = last;
        nb = (s.P - 2 + s.P) % s.P;
        const size_t r = tri(l);
        const double Rl = s.rowR[l];
        const double vbl = s.Vb[l + 1];
        const int nmax = min(l + 1, N - 1);
        double xl[D];
#pragma unroll
        for (int a = 0; a < D; ++a) xl[a] = s.x[idx<D>(s, last, a, l)];
        const int n0 = (band > 0 && !exact) ? max(0, l + 1 - band) / 32 * 32 : 0;
        for (int n = n0 + lane; n <= nmax; n += 32) {
            double pr;
            if (n <= l) {
                // a zero weight (a cycle too costly to contribute) adds exactly 0
                if (!exact && s.Wf[r + n] == 0.0) continue;
                pr = exact ? exp(-beta * (s.V[n] + s.E[r + n] + vbl - VN)) / (l + 1) : s.Wf[r + n] * s.yf[n] * Rl;
            } else {
                pr = 1.0 - s.rowC[l];
            }
#pragma unroll
            for (int a = 0; a < D; ++a) {
                double d = (xs ? xs[(size_t)a * N + n] : s.x[idx<D>(s, first, a, n)]) - xl[a];
                if (s.pbc) d = min_image(d, s.L, s.invL);
                sum[a] += pr * d;
            }
        }
    } else {  // first bead, particle l: sum over q >= l-1
        l = w - N;
        bead = first;
        nb = 1 % s.P;
        const double yl = s.yf[l];
        const double vl = s.V[l];
        double xl[D];
#pragma unroll
        for (int a = 0; a < D; ++a) xl[a] = s.x[idx<D>(s, first, a, l)];
        const int qend = (band > 0 && !exact) ? min(N, l + band) : N;  // q + 1 - l <= band
        for (int q = max(0, l - 1) + lane; q < qend; q += 32) {
            double pr;
            if (q >= l) {
                if (!exact && s.Wf[tri(q) + l] == 0.0) continue;
                pr = exact ? exp(-beta * (vl + s.E[tri(q) + l] + s.Vb[q + 1] - VN)) / (q + 1)
                           : s.Wf[tri(q) + l] * yl * s.rowR[q];
            } else {
                pr = 1.0 - s.rowC[q];
            }
#pragma unroll
            for (int a = 0; a < D; ++a) {
                double d = (xs ? xs[((size_t)D + a) * N + q] : s.x[idx<D>(s, last, a, q)]) - xl[a];
                if (s.pbc) d = min_image(d, s.L, s.invL);
                sum[a] += pr * d;
            }
        }
    }
#pragma unroll
    for (int a = 0; a < D; ++a) sum[a] = warp_sum(sum[a]);
    if (lane == 0 && adjoint) {
        const int side = (bead == first) ? 0 : 1;
        const double c = -vb_bar * s.kappa;
#pragma unroll
        for (int a = 0; a < D; ++a) s.fx[((size_t)side * D + a) * s.ld + l] = c * sum[a];
    } else if (lane == 0) {
        const int side = (bead == first) ? 0 : 1;
#pragma unroll
        for (int a = 0; a < D; ++a) {
            double d = s.x[idx<D>(s, nb, a, l)] - s.x[idx<D>(s, bead, a, l)];
            if (s.pbc) d = min_image(d, s.L, s.invL);
            const double fs = (sum[a] + d) * s.kappa;
            s.fx[((size_t)side * D + a) * s.ld + l] = fs;
            if (accumulate) {
                const size_t o = idx<D>(s, bead, a, l);
                s.f[o] = fs + s.f[o];
            }
        }
    }
}
// primEstimator (:250-279), getDistinctProbability (:222-229) and
// getLongestProbability (:238-240), on request.  The reference evaluates
// primEstimator by a recursion over levels, G[m] = sum_u (G[u] - E[m-1][u])
// exp(-beta (E[m-1][u] + V[u] - V[m])) / m; solved for G[N] it is minus the
// mean energy of the closed cycles,
//   G[N] = - sum_{l,u} p[l][u] E[l][u],
// with the probabilities p[l][u] = Wf[l][u] y_u R_l (u <= l) that
// exch_force_row sums: every entry is independent, where the recursion is a
// chain of N block reductions on one block (a whole pimdb_exchange call at
// N = 777: 8.46 ms with the recursion, 0.35 ms with the sum).
// Each particle is in exactly one cycle, so sum p (l - u + 1) = N; dividing
// by that sum takes out the common rounding of R.
//
// The shares of the rows w0, w0 + nw, ... of one warp: this lane's part of
// sum p E and of sum p (l - u + 1).  `band` as in exch_force_row.
__device__ inline void estimator_rows(const Sys& s, int w0, int nw, int lane, int band, double& pe, double& pn) {
    const int N = s.N;
    const double beta = s.beta_ex, VN = s.V[N];
    const bool exact = s.xflags[0] != 0;
    pe = pn = 0.0;
    for (int l = w0; l < N; l += nw) {
        const size_t r = tri(l);
        const double Rl = s.rowR[l], vbl = s.Vb[l + 1];
        const int n0 = (band > 0 && !exact) ? max(0, l + 1 - band) / 32 * 32 : 0;
        double re = 0.0, rn = 0.0, len = (double)(l + 1 - n0 - lane);
        for (int n = n0 + lane; n <= l; n += 32, len -= 32.0) {
            const double E = s.E[r + n];
            double pr;
            if (exact) {
                pr = exp(-beta * (s.V[n] + E + vbl - VN)) / (l + 1);
            } else {
                const double w = s.Wf[r + n];
                if (w == 0.0) continue;  // a cycle too costly to contribute adds exactly 0
                pr = w * s.yf[n];
            }
            re = fma(pr, E, re);
            rn = fma(pr, len, rn);
        }
        pe = fma(re, exact ? 1.0 : Rl, pe);
        pn = fma(rn, exact ? 1.0 : Rl, pn);
    }
}
// The scalars from the totals of the rows and sum_m E[m][m] (one thread).
__device__ inline void estimator_scalars(const Sys& s, int nbeads, double pe, double pn, double diag) {
    const int N = s.N;
    const double beta = s.beta_ex, VN = s.V[N];
    s.scal[1] = -(pe / pn) * N / nbeads;
    s.scal[2] = exp(-beta * (diag - VN) - lgamma((double)(N + 1)));
    s.scal[3] = exp(-beta * (s.E[tri(N - 1)] - VN));
}
// All of it by one block; `red` holds 32 doubles.
__device__ inline void estimators_block(const Sys& s, int nbeads, double* red) {
    double pe, pn, diag = 0.0;
    estimator_rows(s, threadIdx.x >> 5, blockDim.x >> 5, threadIdx.x & 31, 0, pe, pn);
    for (int m = threadIdx.x; m < s.N; m += blockDim.x) diag += s.E[tri(m) + m];
    pe = block_sum(pe, red);
    pn = block_sum(pn, red);
    diag = block_sum(diag, red);
    if (threadIdx.x == 0) estimator_scalars(s, nbeads, pe, pn, diag);
}

}  // namespace pimdb
