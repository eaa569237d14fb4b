// Feldman-Hirshberg bosonic exchange on the first and last beads.
//
// Reference: BosonicExchange (src/bosonic_exchange/quadratic_bosonic_exchange.cpp)
//   evaluateCycleEnergies :34-61            -> k_exch_energies_rows (below 512
//                                              particles), k_exch_energies_flat
//   evaluateVBn :73-99, evaluateVBackwards :101-128
//                                           -> estimate + weights + solve (below)
//   evaluateConnectionProbabilities :142-157,
//   springForceLastBead / springForceFirstBead :159-215
//                                           -> k_exch_forces (probabilities formed on the fly)
//   primEstimator :250-279 (as a sum over the connection probabilities),
//   getDistinctProbability :222-229,
//   getLongestProbability :238-240          -> k_exch_estimators
//
// Cycle energies are stored packed by row: the reference's E(m, k) (cycle of
// particles m-k+1..m, 1-based) lives at row v = m-1, column u = m-k, offset
// v(v+1)/2 + u, which is exactly the reference's E_kn[m(m+1)/2 - k].
//
// How the recursions are evaluated.  The reference's forward recursion
//   V[m] = -1/beta log( 1/m sum_{u<m} exp(-beta (E[m-1][u] + V[u])) )
// is sequential in m and costs one FP64 exponential per term, which on one
// streaming multiprocessor is far too slow (GB300 runs FP64 at 1/64 of FP32).
// It is evaluated in three passes with the same result in FP64:
//   1. k_exch_estimate / k_exch_estimate_grid (from 512 particles, across
//      SMs): the recursion in FP32 (hardware exp2) in blocks of 32 levels.
//      Gives Vh.
//   2. k_exch_weights_rows, k_exch_weights: every FP64 exponential at once, spread over the GPU:
//      Wf[m-1][u] = exp(-beta (E[m-1][u] + Vh[u] - Vh[m])) / m.
//   3. k_exch_solve: y_0 = 1, y_m = sum_u Wf[m-1][u] y_u (an FP64 triangular
//      solve, multiply-adds only) and V[m] = Vh[m] - log(y_m)/beta exactly.
// Because Vh is within FP32 accuracy of V, every y stays near 1, no term
// over- or underflows and the FP64 result carries the reference's precision.
// If the estimate is ever off by more than 200 kT (not expected; e.g. for
// non-finite input), the solve kernel recomputes the level-by-level FP64
// log-sum-exp in the reference's own order instead.  The backward recursion
// is handled the same way by the second block of each kernel.
// Usually the previous evaluations' potentials (extrapolated linearly) serve
// as Vh and pass 1 is skipped; a solve that fails with them is retried from
// a fresh estimate, in the solving block below the multi-SM solve's size and
// by the phase-1 launches from there on.
// Launches per evaluation below 512 particles: k_exch_energies_rows (the
// energies, a due estimate in its last block, the weights), then
// k_exch_solve_band (pass 3 whole: banded or dense solve, post-processing,
// retry, finish), then k_exch_forces.  From 512 particles the passes run as
// the separate kernels named above, the solve across SMs from 768
// (k_exch_solve_grid) unless the weights are banded.
#include <algorithm>
#include <atomic>

#include "exchange_dev.cuh"
#include "kernels.h"

namespace pimdb {

// Cycle energies: one warp per row.
template <int D>
__global__ void k_exch_energies(Sys s) {
    const int lane = threadIdx.x & 31;
    const int v = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (v >= s.N) return;
    energy_row<D>(s, v, lane);
}

// Cycle energies below the flat form's size, one block per row: the row's
// 32-entry chunks (u = v - 1 - 32 k - lane) are independent but for the
// running carry, so every warp scans its chunks at once; thread 0 then
// forms each chunk's carry from E[v][v] and the chunk totals in the order
// energy_row adds them, and the warps add it.  The terms, the scans and the
// carries are energy_row's, operation for operation: the same bits.  The
// critical path of a row is one chunk instead of all of them.
// The weights follow in the same launch (k_exch_weights' phase-0 work, with
// its band measurement).  With the previous potentials as the estimate, each
// block forms its own row's weights (exch_weight, FP64) from the energies it
// just wrote.  When a fresh estimate is due, the block that finishes last
// runs it (both directions side by side) and then forms every weight with
// double-float exponentials on the FP32 pipe (weights_df_block_f64arg; on one
// SM the FP64 exponentials would take a quarter of a millisecond).  Four blocks per SM
// bound the registers (the rare estimate's arrays would otherwise set them
// for every row).
constexpr int kEnergyRowThreads = 256;
static_assert(kEnergyRowThreads == kWaveThreads, "the estimate runs with the energy kernel's block");
template <int D>
__global__ void __launch_bounds__(kEnergyRowThreads, 4) k_exch_energies_rows(Sys s) {
    extern __shared__ double rsm[];  // scans [N], then the chunks' totals and carries
    __shared__ double wtbl[32];      // exp_tang's table
    const int v = blockIdx.x, N = s.N;
    if (threadIdx.x < 32) wtbl[threadIdx.x] = kExp2Table[threadIdx.x];
    const int fresh = ((volatile int*)s.xflags)[3];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int first = 0, last = s.P - 1;
    const double hk = 0.5 * s.kappa;
    const int nch = (v + 31) / 32;  // chunks of u = v-1 .. 0
    double* scan = rsm;
    double* tot = rsm + N;
    double* carry = tot + nch;
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
    for (int k = warp; k < nch; k += nw) {
        const int base = v - 1 - 32 * k, u = base - lane;
        const double c = u >= 0 ? dist_to_v(u) : 0.0;
        double cu1 = __shfl_up_sync(0xffffffffu, c, 1);
        if (lane == 0) cu1 = dist_to_v(base + 1);  // the previous chunk's last distance
        double term = 0.0;
        if (u >= 0) term = hk * (sepsq<D>(s, last, u, first, u + 1) - cu1 + c);
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const double y = __shfl_up_sync(0xffffffffu, term, o);
            if (lane >= o) term += y;
        }
        if (u >= 0) scan[32 * k + lane] = term;
        const double tk = __shfl_sync(0xffffffffu, term, 31);
        if (lane == 0) tot[k] = tk;
    }
    __syncthreads();
    double* row = s.E + tri(v);
    if (threadIdx.x == 0) {
        double cr = hk * dist_to_v(v);
        row[v] = cr;
        if (v >= 1) s.Et[tri(N - v - 1) + (N - 1 - v)] = cr;
        for (int k = 0; k < nch; ++k) {
            carry[k] = cr;
            cr += tot[k];
        }
    }
    __syncthreads();
    for (int e = threadIdx.x; e < v; e += blockDim.x) {
        const int k = e >> 5, u = v - 1 - e;
        const double val = carry[k] + scan[e];
        row[u] = val;
        // backward node r = N - u depends on node r' = N - 1 - v
        if (u >= 1) s.Et[tri(N - u - 1) + (N - 1 - v)] = val;
    }
    if (!fresh) {
        __syncthreads();  // this row's energies, written by the block
        const double inv = recip_row(v);
        int band = 0;
        for (int u = threadIdx.x; u <= v; u += blockDim.x)
            if (exch_weight(s, v, u, inv, wtbl)) band = max(band, v + 1 - u);
        band = __reduce_max_sync(0xffffffffu, band);
        if ((threadIdx.x & 31) == 0 && band > 0) atomicMax(&s.xflags[kExchBand], band);
    }
    __shared__ int is_last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) is_last = atomicAdd(&s.xflags[kExchRowsCount], 1) == (int)gridDim.x - 1;
    __syncthreads();
    if (!is_last) return;
    __threadfence();
    if (threadIdx.x == 0) {
        s.xflags[kExchRowsCount] = 0;
        s.xflags[7] = !fresh;
        if (fresh) atomicAdd(&s.xflags[kExchFreshCount], 1);
    }
    if (!fresh) return;
    estimate_both(s, reinterpret_cast<float*>(rsm));
    __syncthreads();
    __shared__ dfl::ExpTable etbl;
    fill_exp_table_df(etbl);
    __syncthreads();
    int band = weights_df_block_f64arg(s, etbl, reinterpret_cast<float*>(rsm));
    band = __reduce_max_sync(0xffffffffu, band);
    if ((threadIdx.x & 31) == 0 && band > 0) atomicMax(&s.xflags[kExchBand], band);
}

// Whether the cycle energies of s come from k_exch_energies_rows (which then
// also runs the phase-0 estimate and weights).
static size_t energies_rows_smem(const Sys& s) {
    return std::max(sizeof(double) * ((size_t)s.N + 2 * (((size_t)s.N + 31) / 32) + 2),
                    sizeof(float) * 6 * ((size_t)s.N + 1));  // the estimate of both directions
}
// The kernel's static shared memory (exp_tang's table, the double-float
// exponential table, the last-block flag) counts against the 48 KB that a
// launch gets without opting in to more.
constexpr size_t kRowsStaticSmem = 32 * sizeof(double) + sizeof(dfl::ExpTable) + 64;
static bool energies_by_rows(const Sys& s, const double* work) {
    return !(work && s.eflat) && energies_rows_smem(s) + kRowsStaticSmem <= 48 * 1024;
}

// Cycle energies for large N without a scan per row.  The row recursion
// telescopes: E[v][u] = k/2 (L[v] - L[u] + |xP_v - x1_u|^2) with the prefix
// sums L[w] = sum_{t<w} |x1_{t+1} - xP_t|^2 of the interior links, so every
// entry is independent.  L is kept in double-double (hi, lo): the difference
// of two long prefix sums then keeps the accuracy of the direct sum.
// k_link_prefix (one link per thread) scans blocks of kLinkBlock links and
// wraps the beads' positions into the box, k_link_carry adds the blocks before
// to each block's sums (on one block the whole scan was one SM's FP64 pipe:
// 104 us at N = 4096, 9 + 6 us so), and k_exch_energies_flat writes E and Et.
__device__ __forceinline__ void dd_add(double ah, double al, double bh, double bl, double& h, double& l) {
    const double s = ah + bh;
    const double bb = s - ah;
    double e = (ah - (s - bb)) + (bh - bb);
    e += al + bl;
    h = s + e;
    l = e - (h - s);
}

constexpr int kLinkBlock = 128;
static int link_blocks(int N) { return (N + kLinkBlock - 1) / kLinkBlock; }

// Lh, Ll: exclusive prefix of the link within its block; tot: the blocks' sums.
template <int D>
__global__ void __launch_bounds__(kLinkBlock) k_link_prefix(Sys s, double* __restrict__ Lh, double* __restrict__ Ll,
                                                            double* __restrict__ wrap, double* __restrict__ tot) {
    __shared__ double sh[kLinkBlock / 32], sl[kLinkBlock / 32];
    const int N = s.N, tid = threadIdx.x, w = blockIdx.x * kLinkBlock + tid;
    const int first = 0, last = s.P - 1;
    // positions of beads 1 and P wrapped into [-L/2, L/2): wrap[side][a][N]
    if (w < N)
#pragma unroll
        for (int a = 0; a < D; ++a) {
            double x1 = s.x[idx<D>(s, first, a, w)], xP = s.x[idx<D>(s, last, a, w)];
            if (s.pbc) {
                x1 -= s.L * rint(x1 * s.invL);
                xP -= s.L * rint(xP * s.invL);
            }
            wrap[(size_t)a * N + w] = x1;
            wrap[(size_t)(D + a) * N + w] = xP;
        }
    // inclusive scan of the block's links in double-double: warps, then across
    double ih = w + 1 <= N - 1 ? sepsq<D>(s, last, w, first, w + 1) : 0.0, il = 0.0;
    const int lane = tid & 31, warp = tid >> 5;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const double yh = __shfl_up_sync(0xffffffffu, ih, o), yl = __shfl_up_sync(0xffffffffu, il, o);
        if (lane >= o) dd_add(yh, yl, ih, il, ih, il);
    }
    if (lane == 31) {
        sh[warp] = ih;
        sl[warp] = il;
    }
    __syncthreads();
    double ph = 0.0, pl = 0.0;
    for (int k = 0; k < warp; ++k) dd_add(ph, pl, sh[k], sl[k], ph, pl);
    if (tid == kLinkBlock - 1) dd_add(ph, pl, ih, il, tot[2 * blockIdx.x], tot[2 * blockIdx.x + 1]);
    const double xh = __shfl_up_sync(0xffffffffu, ih, 1), xl = __shfl_up_sync(0xffffffffu, il, 1);
    if (lane > 0) dd_add(ph, pl, xh, xl, ph, pl);
    if (w < N) {
        Lh[w] = ph;
        Ll[w] = pl;
    }
}
__global__ void __launch_bounds__(kLinkBlock) k_link_carry(int N, double* __restrict__ Lh, double* __restrict__ Ll,
                                                           const double* __restrict__ tot) {
    const int w = blockIdx.x * kLinkBlock + threadIdx.x, lane = threadIdx.x & 31;
    // the sum of the blocks before, by every warp alike
    double ch = 0.0, cl = 0.0;
    for (int k = lane; k < (int)blockIdx.x; k += 32) dd_add(ch, cl, tot[2 * k], tot[2 * k + 1], ch, cl);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const double yh = __shfl_xor_sync(0xffffffffu, ch, o), yl = __shfl_xor_sync(0xffffffffu, cl, o);
        dd_add(ch, cl, yh, yl, ch, cl);
    }
    if (w < N) dd_add(ch, cl, Lh[w], Ll[w], Lh[w], Ll[w]);
}

// The lower triangle in tiles of 16 rows and 32 columns (row tiles 2k and
// 2k + 1 have k + 1 column tiles each), row-major: those of the flat energies
// and of the weights, whose second copies (Et, Wb) are packed by column.  The
// transposed entries are written from the registers: staged in shared memory,
// to be written in runs, they kept these blocks off the SMs that the pair
// tiles fill (2 steps of a liquid of 643 particles and 54 beads 1041 us with
// the staging, 866 without; N = 4096 the same).
constexpr int kTileRows = 16, kTileCols = 32, kTileThreads = 128;
constexpr int kTileWarps = kTileThreads / 32, kTilePer = kTileRows / kTileWarps;  // rows per warp
__device__ __forceinline__ void tile_of(int t, int& v0, int& u0) {
    int k = (int)((sqrtf(4.0f * (float)t + 1.0f) - 1.0f) * 0.5f);
    while ((k + 1) * (k + 2) <= t) ++k;
    while (k * (k + 1) > t) --k;
    const int r = t - k * (k + 1), odd = r > k;
    v0 = kTileRows * (2 * k + odd);
    u0 = kTileCols * (r - odd * (k + 1));
}
static int tile_count(int N) {
    const int M = (N + kTileRows - 1) / kTileRows, k = M / 2;
    return k * (k + 1) + (M & 1) * (k + 1);
}
// E and Et from the prefix sums.  Under PBC the image of x1_u nearest to xP_v
// is chosen on FP32 differences: xP_v minus x1_u + L, x1_u or x1_u - L, each
// rounded once per tile; within 1e-6 L of the half-box edge, where FP32 might
// choose the other image, by the FP64 difference.  Bound: the FP64 pipe, 11
// operations an entry (3D): 302 -> 253 us at N = 4096, 19 -> 13 us at N = 777
// against one block per row with the image taken from the FP64 difference.
template <int D>
__global__ void __launch_bounds__(kTileThreads) k_exch_energies_flat(Sys s, const double* __restrict__ Lh,
                                                                     const double* __restrict__ Ll,
                                                                     const double* __restrict__ wrap) {
    const int N = s.N, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int v0, u0;
    tile_of(blockIdx.x, v0, u0);
    const int u = u0 + lane;
    const double hk = 0.5 * s.kappa;
    const float Lf = round_f32(s.L), halfLf = 0.5f * Lf, amb = 1e-6f * Lf;
    double xu[D], xup[D], xum[D];
    float xuf[D];
    double luh = 0.0, lul = 0.0;
#pragma unroll
    for (int a = 0; a < D; ++a) {
        xu[a] = u < N ? wrap[(size_t)a * N + u] : 0.0;
        xuf[a] = round_f32(xu[a]);
        xup[a] = xum[a] = xu[a];
        if (s.pbc) {
            xup[a] += s.L;
            xum[a] -= s.L;
        }
    }
    if (u < N) {
        luh = Lh[u];
        lul = Ll[u];
    }
    // the warp's rows, their values loaded together
    double xv[kTilePer][D], lvh[kTilePer], lvl[kTilePer];
#pragma unroll
    for (int k = 0; k < kTilePer; ++k) {
        const int v = min(v0 + warp + kTileWarps * k, N - 1);
#pragma unroll
        for (int a = 0; a < D; ++a) xv[k][a] = wrap[(size_t)(D + a) * N + v];
        lvh[k] = Lh[v];
        lvl[k] = Ll[v];
    }
#pragma unroll
    for (int k = 0; k < kTilePer; ++k) {
        const int r = warp + kTileWarps * k, v = v0 + r;
        if (v >= N) break;  // rows ascend: uniform in the warp
        double c = 0.0;
#pragma unroll
        for (int a = 0; a < D; ++a) {
            double d;
            if (s.pbc) {
                const float df = round_f32(xv[k][a]) - xuf[a];
                const float over = fabsf(df) - halfLf;
                const double im = over > 0.0f ? (df > 0.0f ? xup[a] : xum[a]) : xu[a];
                d = xv[k][a] - im;
                if (fabsf(over) <= amb) {
                    d = xv[k][a] - xu[a];
                    if (fabs(d) > 0.5 * s.L) d -= copysign(s.L, d);
                }
            } else {
                d = xv[k][a] - xu[a];
            }
            c = a == 0 ? d * d : fma(d, d, c);
        }
        const double e = hk * (((lvh[k] - luh) + (lvl[k] - lul)) + c);
        if (u <= v) s.E[tri(v) + u] = e;
        // backward node r = N - u depends on node r' = N - 1 - v
        if (u >= 1 && u <= v && v < N) s.Et[tri(N - u - 1) + (N - 1 - v)] = e;
    }
}

// Pass 1: block 0 forward, block 1 backward.  Phase 0 skips (early exit)
// when the previous evaluation's exact potentials are still a good estimate
// (xflags[3] == 0) and records in xflags[7] that they were reused; phase 1
// (the retry) runs only when the solve asked for it (xflags[6]).
__global__ void __launch_bounds__(kWaveThreads) k_exch_estimate(Sys s, int phase) {
    if (phase == 0) {
        const int fresh = ((volatile int*)s.xflags)[3];
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            s.xflags[7] = !fresh;
            if (fresh) atomicAdd(&s.xflags[kExchFreshCount], 1);
        }
        if (!fresh) return;
    } else if (((volatile int*)s.xflags)[6] == 0) {
        return;
    }
    extern __shared__ float fsm[];  // 3 (N+1)
    estimate_direction(s, blockIdx.x, fsm);
}

// Pass 1 across SMs, from the flat energies' size: on two blocks it took
// 10.4 ms at N = 4096 and 0.71 ms at N = 777 (here 0.63 and 0.12 ms; 5 us per
// block of nodes).  The schedule is
// k_exch_solve_grid's (below): 32-node blocks go round-robin to `nct` CTAs per
// direction (all resident: cooperative launch); the owner of block j + 1 folds
// block j into it first, from entries loaded while it waited, resolves and
// publishes it (g of its nodes, a fence, a flag), and then folds block j into
// its other rows.  The critical path per block is a flag, one 32 x 32 fold and
// 32 dependent log-sums.  Waits give up after a bounded number of polls
// (ERRB_TIMEOUT).  The estimate itself goes to Vh / Vbh.
__global__ void __launch_bounds__(kGridSolveThreads) k_exch_estimate_grid(Sys s, int phase, float* gsol,
                                                                         unsigned* gflags, int nct) {
    if (phase == 0) {
        const int fresh = ((volatile int*)s.xflags)[3];
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            s.xflags[7] = !fresh;
            if (fresh) atomicAdd(&s.xflags[kExchFreshCount], 1);
        }
        if (!fresh) return;
    } else if (((volatile int*)s.xflags)[6] == 0) {
        return;
    }
    extern __shared__ float esm[];
    __shared__ float gj[32];
    __shared__ int abort_estimate;
    const int dir = blockIdx.x / nct, c = blockIdx.x % nct;
    const EstDir d(s, dir);
    const int nn = d.nn, nb = (nn + 31) / 32, nbmax = (s.N + 1 + 31) / 32;
    const int nown = (nb - c + nct - 1) / nct;  // blocks c, c + nct, ...
    float* gout = gsol + (size_t)dir * (s.N + 1);
    unsigned* flags = gflags + (size_t)dir * nbmax;
    float* mx = esm;               // [nown][32]
    float* sm = esm + nown * 32;   // [nown][32]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int i = tid >> 3, part = tid & 7;  // fold role: row of the block, 4 of its 32 columns
    for (int e = tid; e < nown * 32; e += blockDim.x) {
        mx[e] = -CUDART_INF_F;
        sm[e] = 0.0f;
    }
    if (tid == 0) abort_estimate = 0;
    __syncthreads();
    unsigned ed[32], en[4];  // the block resolved next: its diagonal block (warp 0), its rows against the block before
    auto prefetch = [&](int b) {
        if (warp == 0) est_load_diagonal(d, 32 * b, lane, ed);
        if (b >= 1 && 32 * b + i < nn) est_load_row(d, 32 * b + i, b - 1, part, en);
    };
    auto diag_publish = [&](int b) {  // warp 0 of the owner of block b
        const int n = 32 * b + lane, o = (b / nct) * 32 + lane;
        const float g = est_diagonal(d, 32 * b, lane, n < nn ? mx[o] : 0.0f, n < nn ? sm[o] : 1.0f, ed);
        if (n < nn) {
            gout[n] = g;
            est_store(s, d, n, g);
        }
        __threadfence();
        __syncwarp();
        if (lane == 0) atomicExch(&flags[b], 1u);
    };
#pragma unroll
    for (int q = 0; q < 4; ++q) en[q] = 0u;
    if (c == 0) {
        prefetch(0);
        if (warp == 0) diag_publish(0);
    }
    if (nb > 1 && 1 % nct == c) prefetch(1);
    for (int j = 0; j + 1 < nb; ++j) {
        if (j % nct != c && tid == 0) {  // the owner of block j has it already
            unsigned it = 0;
            while (((volatile unsigned*)flags)[j] == 0u) {
                if (++it > (1u << 22)) {
                    atomicOr(s.err, ERRB_TIMEOUT);
                    abort_estimate = 1;
                    break;
                }
                if (it > 64) __nanosleep(32);
            }
            __threadfence();
        }
        __syncthreads();
        if (abort_estimate) break;
        if (tid < 32) gj[tid] = ((volatile float*)gout)[32 * j + tid];  // j + 1 < nb: a full block
        __syncthreads();
        const int jn = j + 1;
        if (jn % nct == c) {  // the critical path: the next block's rows, then that block
            const bool valid = 32 * jn + i < nn;
            const int o = (jn / nct) * 32 + i;
            est_fold(d, en, gj, part, valid, mx + o, sm + o);
            __syncthreads();
            if (warp == 0) diag_publish(jn);
        }
        for (int r = jn + (c - jn % nct + nct) % nct; r < nb; r += nct) {
            if (r == jn) continue;
            const bool valid = 32 * r + i < nn;
            const int o = (r / nct) * 32 + i;
            unsigned e[4] = {0u, 0u, 0u, 0u};
            if (valid) est_load_row(d, 32 * r + i, j, part, e);
            est_fold(d, e, gj, part, valid, mx + o, sm + o);
        }
        // entries for the next block this CTA resolves, while others work
        if (jn + 1 < nb && (jn + 1) % nct == c) prefetch(jn + 1);
        __syncthreads();
    }
    // the CTA that finishes last clears the flags for the next launch
    __syncthreads();
    if (tid == 0) {
        __threadfence();
        if (atomicAdd(&gflags[2 * nbmax], 1u) == gridDim.x - 1) {
            for (int e = 0; e < 2 * nbmax; ++e) gflags[e] = 0u;
            gflags[2 * nbmax] = 0u;
            __threadfence();
        }
    }
}

// Pass 2: every FP64 exponential at once, one thread per packed entry
// (grid-stride over rows; phase 1 runs only on a retry).  Also records the band
// of the weights (kExchBand: the largest p + 1 - u of a nonzero weight) for the
// banded solve; one atomic per warp.
__global__ void __launch_bounds__(256) k_exch_weights_rows(Sys s, int phase) {
    if (phase == 1 && ((volatile int*)s.xflags)[6] == 0) return;
    __shared__ double tbl[32];
    if (threadIdx.x < 32) tbl[threadIdx.x] = kExp2Table[threadIdx.x];
    __syncthreads();
    int band = 0;
    for (int p = blockIdx.y; p < s.N; p += gridDim.y) {
        const double inv = recip_row(p);
        for (int u = blockIdx.x * blockDim.x + threadIdx.x; u <= p; u += gridDim.x * blockDim.x)
            if (exch_weight(s, p, u, inv, tbl)) band = max(band, p + 1 - u);
    }
    band = __reduce_max_sync(0xffffffffu, band);
    if ((threadIdx.x & 31) == 0 && band > 0) atomicMax(&s.xflags[kExchBand], band);
}
// The same by tiles, for large systems.  An entry whose FP32 argument, with the
// roundings of E and the two potentials added, is below -701 is exactly zero
// (exp_tang's) without any FP64 operation: nearly all of them in a large liquid
// (N = 4096: 245 -> 114 us).  Each thread takes four entries in turn, so below
// kTileWeightsMinN, where that leaves few warps, the row form's one entry a
// thread hides its latencies better, above all beside the pair tiles (steps of
// a liquid, 14 and 24 beads, us, rows / tiles: N = 512 145 / 159 and 157 / 181,
// N = 692 190 / 208 and 206 / 220).  Recursions alone, us, liquid and (no
// weight zero) trap: N = 767 106 / 108 and 225 / 229, N = 1100 175 / 178 and
// 232 / 240, N = 1500 228 / 220 and 307 / 305, N = 4096 553 / 421 and 933 / 813.
// From 1000 particles on the form hardly shows in a step (liquids of 1000, 14
// and 24 beads: 331 / 335 and 455 / 459; dipoles of 1000, 16 and 32 beads 247 /
// 247 and 275 / 277; of 1024 and 32 beads with a cold L2 281 / 276).
constexpr int kTileWeightsMinN = 1024;
__global__ void __launch_bounds__(kTileThreads) k_exch_weights(Sys s, int phase, int tiles) {
    if (phase == 1 && ((volatile int*)s.xflags)[6] == 0) return;
    __shared__ double tbl[32];
    if (threadIdx.x < 32) tbl[threadIdx.x] = kExp2Table[threadIdx.x];
    __syncthreads();
    const int N = s.N, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const double beta = s.beta_ex;
    const float bf = round_f32(beta);
    // whether w = exp(-beta (E + a - b)) / (p + 1) can be other than zero
    auto live = [&](float E, float a, float b) {
        return !(-(E + (a - b)) + 4e-7f * (fabsf(E) + fabsf(a) + fabsf(b)) < -701.0f);
    };
    int band = 0;
    for (int t = blockIdx.x; t < tiles; t += gridDim.x) {
        int p0, u0;
        tile_of(t, p0, u0);
        const int u = u0 + lane;
        const double vu = u < N ? s.Vh[u] : 0.0, vbu = u < N ? s.Vbh[u] : 0.0;
        double E[kTilePer];
#pragma unroll
        for (int k = 0; k < kTilePer; ++k) {
            const int p = p0 + warp + kTileWarps * k;
            E[k] = p < N && u <= p ? s.E[tri(p) + u] : 0.0;
        }
#pragma unroll
        for (int k = 0; k < kTilePer; ++k) {
            const int r = warp + kTileWarps * k, p = p0 + r;
            if (p >= N) break;
            const double vp = s.Vh[p + 1], vbp = s.Vbh[p + 1];
            const float ef = bf * round_f32(E[k]);
            const bool lf = u <= p && live(ef, bf * round_f32(vu), bf * round_f32(vp));
            // backward node r = N - u from node r' = N - 1 - p (u >= 1)
            const bool lb = u <= p && u >= 1 && live(ef, bf * round_f32(vbp), bf * round_f32(vbu));
            double wf = 0.0, wb = 0.0;
            if (__any_sync(0xffffffffu, lf || lb)) {  // the warp's FP64 part, or none of it
                const double inv = recip_row(p);
                if (lf) wf = weight_exp(-beta * (E[k] + vu - vp), tbl) * inv;
                if (lb) wb = weight_exp(-beta * (E[k] + vbp - vbu), tbl) * inv;
                if (!f64_is_zero(wf) || !f64_is_zero(wb)) band = max(band, p + 1 - u);
            }
            if (u <= p) s.Wf[tri(p) + u] = wf;
            if (u >= 1 && u <= p) s.Wb[tri(N - u - 1) + (N - 1 - p)] = wb;
        }
    }
    band = __reduce_max_sync(0xffffffffu, band);
    if (lane == 0 && band > 0) atomicMax(&s.xflags[kExchBand], band);
}

// Pass 3: block 0 forward, block 1 backward.  Phase 0 may not fall back to
// the exact recursion when it reused the previous potentials (xflags[7]); a
// failed solve then leaves xflags[6] set and the phase-1 kernels redo the
// evaluation from a fresh estimate.  With `inline_retry` (smaller systems,
// where the retry's three launches would cost more than its work) the block
// whose solve failed redoes its direction itself: FP32 estimate, weights,
// solve; no phase 1 is launched.  No static shared memory beyond a flag:
// the block has to fit beside the pair kernel's resident blocks.
__global__ void __launch_bounds__(kWaveThreads) k_exch_solve(Sys s, int force_exact, int phase,
                                                             const double* __restrict__ pre, int inline_retry) {
    extern __shared__ double ys[];  // y: N+1, acc: N+1, then 32 for reductions
    __shared__ int last_block;
    __shared__ dfl::ExpTable etbl;  // log y and the row exponentials in double-float
    if (phase == 1 && ((volatile int*)s.xflags)[6] == 0) return;
    if (phase == 0) {
        // k_exch_solve_band post-processed both directions and finished: it
        // set the flag to 2, and each of the two blocks takes one off
        if (threadIdx.x == 0) {
            last_block = ((volatile int*)s.xflags)[kExchBandDone] > 0;
            if (last_block) atomicSub(&s.xflags[kExchBandDone], 1);
        }
        __syncthreads();
        if (last_block) return;
    }
    fill_exp_table_df(etbl);
    __syncthreads();
    if (phase == 1 && blockIdx.x == 0 && threadIdx.x == 0) atomicAdd(&s.xflags[kExchRetryCount], 1);
    const int allow_exact = force_exact || phase == 1 || !((volatile int*)s.xflags)[7];
    const int dir = blockIdx.x;
    const int gave_up = solve_direction(s, dir, force_exact, ys, allow_exact,
                                        pre ? pre + (size_t)dir * (s.N + 1) : nullptr, !inline_retry, &etbl);
    if (gave_up && inline_retry) {
        if (threadIdx.x == 0) atomicAdd(&s.xflags[kExchRetryCount], 1);
        estimate_direction(s, dir, reinterpret_cast<float*>(ys));  // 3 (N+1) floats fit in ys
        __syncthreads();
        weights_direction(s, dir, nullptr);  // CUDA's exp (a rare path)
        __syncthreads();
        solve_direction(s, dir, 0, ys, 1, nullptr, 1, &etbl);
    }
    // The block that finishes second runs solve_finish (threadFenceReduction
    // pattern; no waiting).
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last_block = (atomicAdd(&s.xflags[2], 1) == 1);
    __syncthreads();
    if (!last_block) return;
    __threadfence();
    if (phase == 0 && ((volatile int*)s.xflags)[6]) {
        if (threadIdx.x == 0) s.xflags[2] = 0;  // retry pending: phase 1 finishes
        return;
    }
    solve_finish(s, !force_exact && phase == 0 && ((volatile int*)s.xflags)[7], &etbl);
    if (threadIdx.x == 0) {
        s.xflags[6] = 0;
        s.xflags[kExchBand] = 0;  // the next evaluation's weights measure it anew
        s.xflags[kExchBandLast] = 0;  // not the banded solve's evaluation: full rows
    }
}

// ---------------------------------------------------------------------------
// Pass 3 across SMs for large N.  The triangular solve y_n = sum_{u<n}
// W[n-1][u] y_u costs N^2/2 FP64 multiply-adds per direction, which on the
// one block of k_exch_solve is bound by a single SM's FP64 pipe.  Here 32-row
// blocks go round-robin to `nct` CTAs per direction (all resident: cooperative
// launch).  Block j's owner resolves its diagonal block with warp shuffles
// (its rows then hold the contributions of blocks < j) and publishes y_j
// behind a fence and a flag.  Once y_j is out, the owner of block j + 1 adds
// W[rows of j + 1][block j] y_j to those rows first, from weights loaded
// while it waited, resolves block j + 1 and publishes it; only then does it
// fold y_j into its other rows, as every other CTA does meanwhile (8 threads
// per row, shuffle sums: a fixed order).  The critical path per block is a
// flag, one 32x32 fold and one diagonal block.  Waits give up after a
// bounded number of polls (ERRB_TIMEOUT).  k_exch_solve then post-processes
// y as usual.
__global__ void __launch_bounds__(kGridSolveThreads) k_exch_solve_grid(Sys s, int phase, double* ysol,
                                                                      unsigned* gflags, int nct, int banded) {
    if (phase == 1 && ((volatile int*)s.xflags)[6] == 0) return;
    if (banded && ((volatile int*)s.xflags)[kExchBand] <= kBandMax) return;  // k_exch_solve_band solved it
    extern __shared__ double gsm[];
    __shared__ int abort_solve;
    const int dir = blockIdx.x / nct, c = blockIdx.x % nct;
    const int nn = dir == 0 ? s.N + 1 : s.N;
    const double* __restrict__ W = dir == 0 ? s.Wf : s.Wb;
    double* y = ysol + (size_t)dir * (s.N + 1);
    const int nbmax = (s.N + 1 + 31) / 32;
    unsigned* flags = gflags + (size_t)dir * nbmax;
    const int nb = (nn + 31) / 32;
    const int nown = (nb - c + nct - 1) / nct;  // blocks c, c + nct, ...
    double* acc = gsm;                           // [nown][32]
    double* yj = gsm + (size_t)nown * 32;        // [32]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (int e = tid; e < nown * 32; e += blockDim.x) acc[e] = 0.0;
    if (tid == 0) abort_solve = 0;
    __syncthreads();
    const int i = tid >> 3, part = tid & 7;  // fold role: row of the block, quarter of the columns
    // weights of the block this CTA resolves next, loaded ahead: its
    // diagonal block (warp 0) and W[rows of b][block b - 1]
    double wd[32], wn[4];
    auto prefetch = [&](int b) {
        if (warp == 0) {
            const int n = 32 * b + lane;
#pragma unroll
            for (int t = 0; t < 32; ++t) wd[t] = (n < nn && n >= 1 && t < lane) ? W[tri(n - 1) + 32 * b + t] : 0.0;
        }
        const int n = 32 * b + i;
#pragma unroll
        for (int q = 0; q < 4; ++q) wn[q] = (b >= 1 && n < nn) ? W[tri(n - 1) + 32 * (b - 1) + 4 * part + q] : 0.0;
    };
    auto diag_publish = [&](int b) {  // warp 0 of the owner of block b
        const int n = 32 * b + lane;
        double a = n == 0 ? 1.0 : (n < nn ? acc[(b / nct) * 32 + lane] : 0.0);
#pragma unroll
        for (int t = 0; t < 32; ++t) {
            const double yt = __shfl_sync(0xffffffffu, a, t);
            if (lane > t) a = fma(wd[t], yt, a);
        }
        if (n < nn) y[n] = a;
        __threadfence();
        __syncwarp();
        if (lane == 0) atomicExch(&flags[b], 1u);
    };
    auto fold = [&](int r, int j, bool pre) {  // owned block r += W[rows of r][block j] y_j
        const int n = 32 * r + i;
        double sum = 0.0;
        if (n < nn) {
            if (pre) {
#pragma unroll
                for (int q = 0; q < 4; ++q) sum = fma(wn[q], yj[4 * part + q], sum);
            } else {
                const double* row = W + tri(n - 1) + 32 * j + 4 * part;
#pragma unroll
                for (int q = 0; q < 4; ++q) sum = fma(row[q], yj[4 * part + q], sum);
            }
        }
        sum += __shfl_xor_sync(0xffffffffu, sum, 1);
        sum += __shfl_xor_sync(0xffffffffu, sum, 2);
        sum += __shfl_xor_sync(0xffffffffu, sum, 4);
        if (part == 0 && n < nn) acc[(r / nct) * 32 + i] += sum;
    };
    if (c == 0) {
        prefetch(0);
        if (warp == 0) diag_publish(0);
    }
    if (nb > 1 && 1 % nct == c) prefetch(1);
    for (int j = 0; j + 1 < nb; ++j) {
        if (j % nct != c && tid == 0) {  // the owner of block j has y_j already
            unsigned it = 0;
            while (((volatile unsigned*)flags)[j] == 0u) {
                if (++it > (1u << 22)) {
                    atomicOr(s.err, ERRB_TIMEOUT);
                    abort_solve = 1;
                    break;
                }
                if (it > 64) __nanosleep(32);
            }
            __threadfence();
        }
        __syncthreads();
        if (abort_solve) break;
        if (tid < 32) {
            const int n = 32 * j + tid;
            yj[tid] = n < nn ? ((volatile double*)y)[n] : 0.0;
        }
        __syncthreads();
        const int jn = j + 1;
        const bool mine = jn % nct == c;
        if (mine) {  // the critical path: the next diagonal block's rows, then that block
            fold(jn, j, true);
            __syncthreads();
            if (warp == 0) diag_publish(jn);
        }
        for (int r = jn + (c - jn % nct + nct) % nct; r < nb; r += nct) {
            if (r == jn) continue;
            fold(r, j, false);
        }
        // weights for the next block this CTA resolves, while others work
        if (jn + 1 < nb && (jn + 1) % nct == c) prefetch(jn + 1);
        __syncthreads();
    }
    // the CTA that finishes last clears the flags for the next launch
    __syncthreads();
    if (tid == 0) {
        __threadfence();
        if (atomicAdd(&gflags[2 * nbmax], 1u) == gridDim.x - 1) {
            for (int e = 0; e < 2 * nbmax; ++e) gflags[e] = 0u;
            gflags[2 * nbmax] = 0u;
            __threadfence();
        }
    }
}

// ---------------------------------------------------------------------------
// Pass 3 when the weights are banded.  A weight is exactly zero when its
// cycle costs beta_ex E > 700 (the exponential's result is returned as 0):
// at liquid-helium densities and temperatures every cycle of more than a
// dozen or so particles, so node n depends only on nodes n - band .. n - 1
// with a band far below N.  k_exch_weights records the band of the current
// evaluation; when it is at most kBandMax (two 32-row blocks) this kernel
// solves each direction on one CTA: block b's rows take the two previous
// blocks' y from shared memory (all threads, 8 columns each), then warp 0
// resolves the diagonal block by shuffles, while warps 1-7 stage the next
// block's weights into the other half of a double buffer.  No flags and no
// inter-CTA waits; y lands in ysol as from the dense solves, which step
// aside (their `banded` argument) and stay the general path.
// `standalone` (below the multi-SM solve's size): this kernel is the whole
// pass 3.  A band above kBandMax is solved densely on the same CTA
// (blocked_solve), a reused estimate that fails is redone from a fresh one
// in the block (k_exch_solve's in-block retry), and the CTA that finishes
// second runs solve_finish; no other solve kernel is launched.
// solve_direction's post-processing of an inexact solve (y in shared memory),
// with one pass over the nodes and one barrier: V or V_backwards, yf / yb and
// the direction's flags.  Returns 1 (block-uniform, the flags untouched) where
// the estimate proves unusable.  `word`: shared scratch.
__device__ __forceinline__ int finish_direction(const Sys& s, int dir, const double* ys, const dfl::ExpTable& et,
                                                int* word) {
    const int N = s.N, tid = threadIdx.x, bd = blockDim.x;
    if (tid == 0) *word = 0;
    __syncthreads();
    const double* Vh = dir == 0 ? s.Vh : s.Vbh;
    double* V = dir == 0 ? s.V : s.Vb;
    double* yo = dir == 0 ? s.yf : s.yb;
    int flags = 0;  // 1 unusable, 2 thirty kT off, 4 not finite
    // (m = 0 of direction 0 is y = 1, V = Vh: left to the thread below, so that
    // N = bd nodes stay one pass)
    for (int m = tid + 1; m < N + (dir == 0); m += bd) {
        const double y = ys[dir == 0 ? m : N - m];
        const double ly = log_df(y, et);
        const double v = Vh[m] - ly * s.inv_beta_ex;
        if (!(y > 0.0) || !(fabs(ly) < kExactLogY)) flags |= 1;
        if (!(fabs(ly) < kRefreshLogY)) flags |= 2;
        if (!isfinite(v)) flags |= 4;
        yo[m] = y;
        V[m] = v;
    }
    if (tid == bd - 1) {
        V[dir == 0 ? 0 : N] = dir == 0 ? Vh[0] : 0.0;
        yo[dir == 0 ? 0 : N] = 1.0;
    }
    if (flags) atomicOr(word, flags);
    __syncthreads();
    flags = *word;
    __syncthreads();
    if (flags & 1) return 1;
    if (tid == 0) {
        s.xflags[dir] = 0;
        s.xflags[4 + dir] = flags >> 1;
        if (flags & 4) atomicOr(s.err, ERRB_NONFINITE_VB);
    }
    return 0;
}
// solve_finish with every load issued at once: node m's row factors and next
// estimate are one thread's.
__device__ __forceinline__ void finish_both(const Sys& s, int extrapolate, const dfl::ExpTable& et) {
    const int N = s.N, tid = threadIdx.x;
    const double beta = s.beta_ex;
    const double VN = __ldcg(s.V + N);
    const int off = __ldcg(s.xflags + 4) | __ldcg(s.xflags + 5);
    const int order = s.Vp ? __ldcg(s.xflags + kExchOrder) : 1;
    auto estimate = [&](int m, double v, double vb, double p, double pb) {
        const bool ext = s.Vp && extrapolate && isfinite(p) && isfinite(pb);
        s.Vh[m] = ext ? 2.0 * v - p : v;
        s.Vbh[m] = ext ? 2.0 * vb - pb : vb;
        if (s.Vp) {
            s.Vp[m] = v;
            s.Vp[N + 1 + m] = vb;
        }
    };
    const bool old = s.Vp && extrapolate;
    // node 0 has no row factors: beside the others, so that N = blockDim.x
    // nodes stay one pass (with the line in finish_direction: recursions of
    // N = 256 43.0 -> 40.8 us)
    double v0 = 0.0, p0 = 0.0, pb0 = 0.0;
    if (tid == 0) {
        v0 = __ldcg(s.V);
        if (old) {
            p0 = s.Vp[0];
            pb0 = s.Vp[N + 1];
        }
    }
    for (int m = tid + 1; m <= N; m += blockDim.x) {
        const double v = __ldcg(s.V + m), vb = __ldcg(s.Vb + m), vh = s.Vh[m];
        const double p = old ? s.Vp[m] : v, pb = old ? s.Vp[N + 1 + m] : vb;
        s.rowR[m - 1] = exp_df(-beta * (vh + vb - VN), et);
        s.rowC[m - 1] = exp_df(-beta * (v + vb - VN), et);
        estimate(m, v, vb, p, pb);
    }
    if (tid == 0) estimate(0, v0, 0.0, p0, pb0);
    __syncthreads();
    if (tid == 0) {
        s.xflags[2] = 0;
        s.xflags[3] = (off & 2) || ((off & 1) && order);
        if (s.Vp) s.xflags[kExchOrder] = extrapolate;
        s.Vb[0] = VN;  // V_backwards[0] = V[N] (:127)
        s.scal[0] = VN;
    }
}

__device__ __noinline__ void band_standalone_tail(const Sys& s, int dir, double* ys, const dfl::ExpTable& etbl,
                                                  int band, bool dense, int* last_band) {
    const int tid = threadIdx.x;
    const int allow_exact = !((volatile int*)s.xflags)[7];  // the estimate was fresh
    int retried = 0;
    if (finish_direction(s, dir, ys, etbl, last_band)) {
        if (allow_exact) {
            solve_direction(s, dir, 0, ys, 1, ys, 0, &etbl);
        } else {
            if (tid == 0) atomicAdd(&s.xflags[kExchRetryCount], 1);
            estimate_direction(s, dir, reinterpret_cast<float*>(ys));  // 3 (N+1) floats fit in ys
            __syncthreads();
            weights_direction(s, dir, nullptr);  // CUDA's exp (a rare path)
            __syncthreads();
            solve_direction(s, dir, 0, ys, 1, nullptr, 1, &etbl);
            retried = 1;
        }
    }
    __syncthreads();
    if (tid == 0) {
        __threadfence();  // after the block's barrier: its results before the count
        // 1 per direction, 16 per direction that was redone
        const int mine = retried ? 16 : 1;
        const int prev = atomicAdd(&s.xflags[kExchBandCount], mine);
        *last_band = prev == 0 ? 0 : 1 + (((prev + mine) >> 4) ? 2 : 0);
    }
    __syncthreads();
    if (*last_band == 0) return;
    __threadfence();
    finish_both(s, *last_band != 3 && !allow_exact, etbl);
    if (tid == 0) {
        s.xflags[6] = 0;
        // full exterior-force rows after a dense solve or a redone direction
        s.xflags[kExchBandLast] = (dense || *last_band == 3) ? 0 : band;
        s.xflags[kExchBand] = 0;  // the next evaluation's weights measure it anew
        s.xflags[kExchBandCount] = 0;
    }
}

// The banded solve by FP32 elimination with FP64 residuals (bands up to 24).
// One warp issues an FP64 instruction every 64 cycles and a dependent
// multiply-add takes 65 (measured), so the chain over the nodes in FP64 costs
// 111 cycles a node whatever its arrangement.  Here each 32-node block's
// unit lower triangle (I - L) is inverted in FP32, all blocks side by side
// (one warp each: inv = (I - L)^-1 and T = inv U with U the rows' weights on
// the previous block's last cw >= band nodes), after which a right-hand side
// is solved by a product with inv per block (side by side) and one cw-term
// sum per block in sequence, e_b = inv rho_b + T e_{b-1}: 330 cycles a
// block of 32 nodes.  y starts at 0 with rho the unit vector; every further
// round takes the residual rho = W y - y in FP64 (all nodes side by side) and
// adds the correction to y in FP64.  What a round leaves is FP32's rounding
// along the chain of the correction it adds (some 1e-5 of it), so after one
// below 1e-10, in general the third or fourth, the error is that of an FP64
// residual: V differs from extended precision as much as with the substitution
// (N = 2016 to 4096, six temperatures: 1e-11 to 2e-10 kT).  Gives up (false;
// block-uniform) where y leaves [1e-20, 1e20], so that corrections of 1e-16
// still are FP32 numbers, or does not converge.
// `Ls`: kBandThreads / 32 x 1024 floats; `fs`: 32 nb floats; `store`: nb
// blocks of T [32][cw + 1] and inv [32][36].
constexpr int kBandWarps = kBandThreads / 32;
// The band it takes, and the blocks from which it is the faster form: its code
// is long and runs once, so few blocks pay more for fetching it than they save
// (steps of N = 256, 9 blocks, and N = 1024, 33 blocks, 2-3% slower with it;
// N = 4096, 129 blocks, 8.21 -> 7.82 ms for 4 steps).  Recursions, us,
// substitution / refined, at bands of 28, 24, 19 and 13: N = 2016 298 / 309,
// 296 / 285, 291 / 272, 287 / 260; N = 2450 352 / 384, 348 / 296, 347 / 293,
// 340 / 278; N = 3100 435 / 443, 431 / 432, 426 / 412, 419 / 350.
constexpr int kBandRefined = 24;
constexpr int kBandRefinedMin = 64;
constexpr int kBandStore = 32 * 25 + 32 * 36;  // floats per block at most (behind ysol)
// A double rounded to float by bit patterns, 0 below 2^-126 and infinite above
// a float's range (the conversion instruction takes the FP64 pipe for 128
// cycles a warp).
__device__ __forceinline__ float f32_of(double x) {
    const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x), e = (hi >> 20) & 0x7ffu;
    unsigned q = ((e - 896u) << 23 | (hi & 0xfffffu) << 3 | lo >> 29) + ((lo >> 28) & 1u);
    if (e <= 896u) q = 0u;
    if (e >= 1151u) q = 0x7f800000u | (e == 0x7ffu ? (hi & 0xfffffu) | lo : 0u);
    return __uint_as_float(q | (hi & 0x80000000u));
}
// e_b = inv rho_b + T e_{b-1} over the blocks, by one warp (lane = row): fs
// holds inv rho_b and receives e_b.  The next block's T is loaded, and the one
// six blocks on prefetched, while this one is summed.
template <int CW>
__device__ __forceinline__ void band_sequence(int nb, float* fs, const float* store, int lane) {
    constexpr int ldt = CW + 1, per = 32 * ldt + 32 * 36;
    float e = fs[lane], next[CW];
    auto fetch = [&](int b) {
#pragma unroll
        for (int c = 0; c < CW; ++c) next[c] = store[(size_t)b * per + lane * ldt + c];
    };
    fetch(1);
    for (int b = 1; b < nb; ++b) {
        float T[CW], s[4] = {fs[32 * b + lane], 0.0f, 0.0f, 0.0f};
#pragma unroll
        for (int c = 0; c < CW; ++c) T[c] = next[c];
        if (b + 6 < nb)
            asm volatile("prefetch.global.L1 [%0];" ::"l"(store + (size_t)(b + 6) * per + lane * ldt));
        if (b + 1 < nb) fetch(b + 1);
#pragma unroll
        for (int c = 0; c < CW; ++c) s[c & 3] = fmaf(T[c], __shfl_sync(0xffffffffu, e, 32 - CW + c), s[c & 3]);
        e = (s[0] + s[1]) + (s[2] + s[3]);
        fs[32 * b + lane] = e;
    }
}
__device__ __noinline__ bool band_refined(const double* __restrict__ W, int nn, int band, double* ys, float* fs,
                                          float* Ls, float* store) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nb = (nn + 31) / 32, cw = (band + 7) & ~7, ldt = cw + 1, per = 32 * ldt + 32 * 36;
    for (int b = warp; b < nb; b += kBandWarps) {
        float* L = Ls + warp * 1024;
        float T[32], I[32];
        // row r's weights on the 32 nodes before it, one load a row; those of
        // this block go to L, those of the previous block to the lane of
        // their column
#pragma unroll
        for (int r0 = 0; r0 < 32; r0 += 16) {
            double w[16];
#pragma unroll
            for (int q = 0; q < 16; ++q) {
                const int m = 32 * b + r0 + q, c = m - 32 + lane;
                w[q] = m < nn && c >= 0 && lane >= 32 - band ? W[tri(m - 1) + c] : 0.0;
            }
#pragma unroll
            for (int q = 0; q < 16; ++q) {
                const int r = r0 + q;
                const float v = f32_of(w[q]);
                const float t = __shfl_sync(0xffffffffu, v, (lane - r) & 31);
                T[r] = lane >= r ? t : 0.0f;
                if (lane + r >= 32) L[r * 32 + lane + r - 32] = v;
            }
        }
        __syncwarp();
        // rows in order; lane = column (of the previous block for T, of this one for inv)
#pragma unroll
        for (int r = 0; r < 32; ++r) {
            float t[4] = {T[r], 0.0f, 0.0f, 0.0f}, i[4] = {lane == r ? 1.0f : 0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
            for (int q = 0; q < r; q += 4) {
                const float4 l = *reinterpret_cast<const float4*>(L + r * 32 + q);  // columns below r are used
                t[0] = fmaf(l.x, T[q], t[0]);
                i[0] = fmaf(l.x, I[q], i[0]);
                if (q + 1 < r) {
                    t[1] = fmaf(l.y, T[q + 1], t[1]);
                    i[1] = fmaf(l.y, I[q + 1], i[1]);
                }
                if (q + 2 < r) {
                    t[2] = fmaf(l.z, T[q + 2], t[2]);
                    i[2] = fmaf(l.z, I[q + 2], i[2]);
                }
                if (q + 3 < r) {
                    t[3] = fmaf(l.w, T[q + 3], t[3]);
                    i[3] = fmaf(l.w, I[q + 3], i[3]);
                }
            }
            T[r] = (t[0] + t[1]) + (t[2] + t[3]);
            I[r] = (i[0] + i[1]) + (i[2] + i[3]);
        }
        float* st = store + (size_t)b * per;
#pragma unroll
        for (int r = 0; r < 32; ++r) {
            if (lane >= 32 - cw) st[r * ldt + lane - (32 - cw)] = T[r];
            st[32 * ldt + r * 36 + lane] = I[r];
        }
        __syncwarp();  // the next block overwrites L
    }
    for (int m = tid; m < nn; m += kBandThreads) ys[m] = 0.0;
    __syncthreads();
    for (int round = 0; round < 6; ++round) {
        for (int m = tid; m < 32 * nb; m += kBandThreads) {
            double r = m == 0 ? 1.0 : 0.0;
            if (round > 0 && m < nn) {
                const double* row = W + (m >= 1 ? tri(m - 1) : 0);
                double r1 = -ys[m];
                int c = max(0, m - band);
                if ((m - c) & 1) {
                    r = fma(row[c], ys[c], r);
                    ++c;
                }
#pragma unroll 8
                for (; c < m; c += 2) {
                    r = fma(row[c], ys[c], r);
                    r1 = fma(row[c + 1], ys[c + 1], r1);
                }
                r += r1;
            }
            fs[m] = f32_of(r);
        }
        __syncthreads();
        for (int b = warp; b < nb; b += kBandWarps) {
            const float4* inv = reinterpret_cast<const float4*>(store + (size_t)b * per + 32 * ldt + lane * 36);
            const float rho = fs[32 * b + lane];
            float z[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
            for (int t = 0; t < 8; ++t) {
                const float4 v = inv[t];
                z[0] = fmaf(v.x, __shfl_sync(0xffffffffu, rho, 4 * t), z[0]);
                z[1] = fmaf(v.y, __shfl_sync(0xffffffffu, rho, 4 * t + 1), z[1]);
                z[2] = fmaf(v.z, __shfl_sync(0xffffffffu, rho, 4 * t + 2), z[2]);
                z[3] = fmaf(v.w, __shfl_sync(0xffffffffu, rho, 4 * t + 3), z[3]);
            }
            fs[32 * b + lane] = (z[0] + z[1]) + (z[2] + z[3]);
        }
        __syncthreads();
        if (warp == 0) {
            if (cw == 8) band_sequence<8>(nb, fs, store, lane);
            else if (cw == 16) band_sequence<16>(nb, fs, store, lane);
            else band_sequence<24>(nb, fs, store, lane);
        }
        __syncthreads();
        int more = 0, bad = 0;
        for (int m = tid; m < nn; m += kBandThreads) {
            const float e = fs[m];
            const double y = ys[m] + f32_to_f64(e);
            const float yf = fabsf(f32_of(y));
            ys[m] = y;
            if (!(fabsf(e) <= 1e-10f * yf)) more = 1;
            if (!(yf >= 1e-20f && yf <= 1e20f)) bad = 1;
        }
        if (__syncthreads_or(bad)) return false;
        if (!__syncthreads_or(more)) return true;
    }
    return false;
}

__global__ void __launch_bounds__(kBandThreads) k_exch_solve_band(Sys s, int phase, double* ysol, int standalone) {
    if (phase == 1 && ((volatile int*)s.xflags)[6] == 0) return;
    const int band = ((volatile int*)s.xflags)[kExchBand];
    const bool dense = band > kBandMax;
    if (dense && !standalone) return;  // the dense solve runs instead
    extern __shared__ double bsm[];
    __shared__ double accb[32];
    __shared__ dfl::ExpTable etbl;
    __shared__ int last_band;
    const int dir = blockIdx.x;
    const int nn = dir == 0 ? s.N + 1 : s.N;
    const double* __restrict__ W = dir == 0 ? s.Wf : s.Wb;
    double* y = ysol + (size_t)dir * (s.N + 1);
    const int nnpad = (nn + 1) & ~1;
    double* ys = bsm;                    // [nn]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nb = (nn + 31) / 32, nbmax = (s.N + 1 + 31) / 32;
    float* fs = reinterpret_cast<float*>(bsm + nnpad);       // [32 nb]
    float* Ls = fs + 32 * nbmax;                             // band_refined's rows
    double* wdiag = reinterpret_cast<double*>(Ls);  // [2][32][32]: block b's diagonal block, row-major
    double* wfold = wdiag + 2 * 1024;    // [2][32][64]: block b's rows, columns 32b - 64 .. 32b - 1
    // the exponential's table beside the first loads (used after barriers)
    if (tid >= kBandThreads - 256) {
        const int j = tid - (kBandThreads - 256);
        float h, l;
        split_f32(kExp2Table256[j], h, l);
        const dfl::df n = dfl::fast_two_sum(h, l);
        etbl.hi[j] = n.hi;
        etbl.lo[j] = n.lo;
    }
    bool solved = false;
    if (band <= kBandRefined && nb >= kBandRefinedMin) {
        float* store = reinterpret_cast<float*>(ysol + 2 * ((size_t)s.N + 1)) + (size_t)dir * nbmax * kBandStore;
        solved = band_refined(W, nn, band, ys, fs, Ls, store);
        if (solved)
            for (int m = tid; m < nn; m += blockDim.x) y[m] = ys[m];
        __syncthreads();
    }
    // Threads t0.. stage block b's weights: row r of the block needs columns
    // 32b - 64 .. 32b + r - 1 of its packed row (contiguous), taken as one
    // row-major index e = 96 r + q (q < 64: fold, else diagonal) so that a
    // warp's loads are coalesced.  Every load of a thread is issued before
    // any store: one L2 round trip per block rather than one per element.
    constexpr int kStagePer = (32 * 96 + (kBandThreads - 32) - 1) / (kBandThreads - 32);
    auto stage = [&](int b, int t0, int nt) {
        double* d = wdiag + (b & 1) * 1024;
        double* f = wfold + (b & 1) * 2048;
        double v[kStagePer];
#pragma unroll
        for (int k = 0; k < kStagePer; ++k) {
            const int e = tid - t0 + k * nt;
            const int r = e / 96, q = e - 96 * r, m = 32 * b + r;
            const int c = q < 64 ? 32 * b - 64 + q : 32 * b + (q - 64);
            const bool in = e < 32 * 96 && m < nn && m >= 1 && (q < 64 ? c >= 0 : q - 64 < r);
            v[k] = in ? W[tri(m - 1) + c] : 0.0;
        }
#pragma unroll
        for (int k = 0; k < kStagePer; ++k) {
            const int e = tid - t0 + k * nt;
            if (e < 32 * 96) {
                const int r = e / 96, q = e - 96 * r;
                if (q < 64) f[r * 64 + q] = v[k];
                else d[r * 32 + (q - 64)] = v[k];
            }
        }
    };
    if (dense) {
        blocked_solve(W, nn, ys, wdiag);  // accumulators in the (unused) staging buffers
        for (int m = tid; m < nn; m += blockDim.x) y[m] = ys[m];
        __syncthreads();
    }
    if (!dense && !solved) stage(0, 0, blockDim.x);
    __syncthreads();
    const int i = tid >> 3, part = tid & 7;  // fold role (threads below 256): row of the block, 8 of its 64 columns
    const int dband = dense ? 32 : band;  // the diagonal chain's reach
    for (int b = 0; b < (dense || solved ? 0 : nb); ++b) {
        const double* f = wfold + (b & 1) * 2048;
        double sum = 0.0;
        // columns more than `band` before the block's first row hold exact
        // zero weights: no multiply-add for them
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const int col = 8 * part + q, c = 32 * b - 64 + col;
            if (i < 32 && c >= 0 && col >= 64 - band) sum = fma(f[i * 64 + col], ys[c], sum);
        }
        sum += __shfl_xor_sync(0xffffffffu, sum, 1);
        sum += __shfl_xor_sync(0xffffffffu, sum, 2);
        sum += __shfl_xor_sync(0xffffffffu, sum, 4);
        if (part == 0 && i < 32) accb[i] = sum;
        __syncthreads();
        if (warp == 0) {
            const double* d = wdiag + (b & 1) * 1024;
            const int m = 32 * b + lane;
            double a = m == 0 ? 1.0 : (m < nn ? accb[lane] : 0.0);
            // lanes more than `band` below t hold exact zero weights for t:
            // only the band's lanes issue the multiply-add
#pragma unroll
            for (int t = 0; t < 32; ++t) {
                const double yt = __shfl_sync(0xffffffffu, a, t);
                if (lane > t && lane - t <= dband) a = fma(d[lane * 32 + t], yt, a);
            }
            if (m < nn) {
                ys[m] = a;
                y[m] = a;
            }
        } else if (b + 1 < nb) {
            stage(b + 1, 32, blockDim.x - 32);
        }
        __syncthreads();
    }
    // The post-processing of k_exch_solve for this direction, from y in
    // shared memory (no exact fallback here: a direction that would need one
    // or a fresh estimate leaves the whole evaluation to k_exch_solve).  The
    // CTA that finishes second runs solve_finish when both directions
    // succeeded and marks the evaluation done.
    if (phase != 0) return;
    if (standalone) {
        band_standalone_tail(s, dir, ys, etbl, band, dense, &last_band);
        return;
    }
    const int gave_up = finish_direction(s, dir, ys, etbl, &last_band);
    if (tid == 0) {
        __threadfence();  // after the block's barrier: its results before the count
        // count 2 per direction that succeeded, 1 per direction that gave up
        const int prev = atomicAdd(&s.xflags[kExchBandCount], gave_up ? 1 : 2);
        last_band = prev > 0 ? (prev + (gave_up ? 1 : 2)) : 0;
    }
    __syncthreads();
    if (last_band == 0) return;
    __threadfence();
    if (last_band == 4) {
        finish_both(s, ((volatile int*)s.xflags)[7], etbl);
        if (tid == 0) {
            s.xflags[kExchBandLast] = s.xflags[kExchBand];
            s.xflags[kExchBand] = 0;  // the next evaluation's weights measure it anew
            s.xflags[kExchBandDone] = 2;  // one for each block of k_exch_solve
        }
    }
    if (tid == 0) s.xflags[kExchBandCount] = 0;
}

bool banded_solve_fits(const Sys& s) { return s.N + 1 <= kBandMaxN; }

static int band_blocks(const Sys& s) { return (s.N + 1 + 31) / 32; }
// Floats of band_refined's store behind ysol (both directions).
static size_t band_store_floats(const Sys& s) {
    return band_blocks(s) < kBandRefinedMin || !banded_solve_fits(s) ? 0 : 2 * (size_t)band_blocks(s) * kBandStore;
}
size_t banded_solve_smem(const Sys& s) {
    const size_t fp64 = sizeof(double) * (2 * 1024 + 2 * 2048);
    const size_t refined = band_blocks(s) < kBandRefinedMin ? 0 : sizeof(float) * kBandWarps * 1024;
    return sizeof(double) * (((size_t)s.N + 2) & ~(size_t)1) + sizeof(float) * 32 * (size_t)band_blocks(s) +
           std::max(refined, fp64);
}


// Exterior spring forces: one warp per row (bead P) or column (bead 1).
template <int D>
__global__ void k_exch_forces(Sys s, int accumulate, int adjoint, double vb_bar) {
    const int lane = threadIdx.x & 31;
    const int w = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (w >= 2 * s.N) return;
    exch_force_row<D>(s, w, lane, accumulate, nullptr, adjoint, vb_bar, ((volatile int*)s.xflags)[kExchBandLast]);
}

// The estimators, rows spread over the GPU: each block writes its totals to
// its slot of Sys::epart and the block that finishes last adds the slots in
// order (no waiting; deterministic).  One warp per row at a time, 16 bytes
// read per packed entry within the band.
__global__ void __launch_bounds__(kEstimatorThreads) k_exch_estimators(Sys s, int nbeads) {
    __shared__ double red[32];
    __shared__ int is_last;
    const int nw = kEstimatorThreads / 32, tid = threadIdx.x;
    double pe, pn, diag = 0.0;
    estimator_rows(s, blockIdx.x * nw + (tid >> 5), gridDim.x * nw, tid & 31,
                   ((volatile int*)s.xflags)[kExchBandLast], pe, pn);
    pe = block_sum(pe, red);
    pn = block_sum(pn, red);
    if (tid == 0) {
        s.epart[2 * blockIdx.x] = pe;
        s.epart[2 * blockIdx.x + 1] = pn;
        __threadfence();
        is_last = atomicAdd(&s.xflags[kExchRowsCount], 1) == (int)gridDim.x - 1;
    }
    __syncthreads();
    if (!is_last) return;
    __threadfence();
    pe = pn = 0.0;
    for (int k = tid; k < (int)gridDim.x; k += kEstimatorThreads) {
        pe += ((volatile double*)s.epart)[2 * k];
        pn += ((volatile double*)s.epart)[2 * k + 1];
    }
    for (int m = tid; m < s.N; m += kEstimatorThreads) diag += s.E[tri(m) + m];
    pe = block_sum(pe, red);
    pn = block_sum(pn, red);
    diag = block_sum(diag, red);
    if (tid == 0) {
        estimator_scalars(s, nbeads, pe, pn, diag);
        s.xflags[kExchRowsCount] = 0;
    }
}

// The exchange kernels that spread over the GPU take the largest shared-memory
// carveout.  An SM runs all its resident blocks under one carveout, so a kernel
// that prefers a smaller one (more L1) could start only on SMs without
// pair-tile blocks, and the pair tiles' blocks could not start beside it:
// launched first in a step graph, the exchange would hold back part of the pair
// kernel.  k_exch_solve_band has two blocks and SMs of its own
// (launch_solve_band), and k_exch_estimators comes last on its stream: with it
// listed too, observables of 100 to 692 particles took the same time.
// Attributes belong to the current device: they are set once per device (a
// bit per device id below 64, every call above), and two host threads that
// set them at once only repeat the same cheap calls.
static std::atomic<unsigned long long> g_carveout_devices{0};

static void exchange_carveouts() {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) {
        cudaGetLastError();
        return;
    }
    const unsigned long long bit = dev >= 0 && dev < 64 ? 1ull << dev : 0ull;
    if (bit && (g_carveout_devices.load(std::memory_order_acquire) & bit)) return;
    const void* k[] = {(const void*)k_exch_energies<1>, (const void*)k_exch_energies<2>,
                       (const void*)k_exch_energies<3>, (const void*)k_exch_energies_rows<1>,
                       (const void*)k_exch_energies_rows<2>, (const void*)k_exch_energies_rows<3>, (const void*)k_link_prefix<1>,
                       (const void*)k_link_prefix<2>, (const void*)k_link_prefix<3>, (const void*)k_link_carry,
                       (const void*)k_exch_energies_flat<1>, (const void*)k_exch_energies_flat<2>,
                       (const void*)k_exch_energies_flat<3>, (const void*)k_exch_estimate, (const void*)k_exch_estimate_grid,
                       (const void*)k_exch_weights, (const void*)k_exch_weights_rows, (const void*)k_exch_solve, (const void*)k_exch_solve_grid,
                       (const void*)k_exch_forces<1>, (const void*)k_exch_forces<2>, (const void*)k_exch_forces<3>};
    for (const void* f : k)
        cudaFuncSetAttribute(f, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
    if (bit) g_carveout_devices.fetch_or(bit, std::memory_order_acq_rel);
}

int exchange_flat_default(int N) { return N >= kFlatEnergiesMinN ? 1 : 0; }

// A launch gets 48 KB of shared memory without opting in, static and
// dynamic together.  The kernels here hold up to about 2.3 KB of static
// shared memory (their exponential tables), so a dynamic size within
// kSmemOptInMargin of 48 KB opts in as well; opting in when the default
// would have done is harmless.
constexpr size_t kSmemOptInMargin = 8 * 1024;
static void opt_in_smem(const void* k, size_t dyn) {
    if (dyn + kSmemOptInMargin > 48 * 1024) cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dyn);
}

// The work array of the prefix-sum energies (any N: Sys::eflat chooses): the
// prefix sums, the wrapped positions, the blocks' sums.
size_t exchange_energy_doubles(const Sys& s, int D) { return (size_t)(2 + 2 * D) * s.N + 2 * (size_t)link_blocks(s.N); }

template <int D>
static void flat_launch(const Sys& s, double* work, cudaStream_t st) {
    const int nb = link_blocks(s.N);
    double* Lh = work;
    double* Ll = work + s.N;
    double* wrap = work + 2 * (size_t)s.N;
    double* tot = wrap + (size_t)2 * D * s.N;
    k_link_prefix<D><<<nb, kLinkBlock, 0, st>>>(s, Lh, Ll, wrap, tot);
    if (nb > 1) k_link_carry<<<nb, kLinkBlock, 0, st>>>(s.N, Lh, Ll, tot);
    k_exch_energies_flat<D><<<tile_count(s.N), kTileThreads, 0, st>>>(s, Lh, Ll, wrap);
}

int launch_exchange_energies(const Sys& s, int D, cudaStream_t st, double* work) {
    exchange_carveouts();
    if (work && s.eflat) {
        if (D == 1) flat_launch<1>(s, work, st);
        else if (D == 2) flat_launch<2>(s, work, st);
        else flat_launch<3>(s, work, st);
        return 0;
    }
    // one block per row; scans [N] and two chunk arrays in shared memory
    // (or the 6 (N + 1) floats of both directions' estimate)
    const size_t rs = energies_rows_smem(s);
    if (energies_by_rows(s, work)) {
        if (D == 1) k_exch_energies_rows<1><<<s.N, kEnergyRowThreads, rs, st>>>(s);
        else if (D == 2) k_exch_energies_rows<2><<<s.N, kEnergyRowThreads, rs, st>>>(s);
        else k_exch_energies_rows<3><<<s.N, kEnergyRowThreads, rs, st>>>(s);
        return 1;
    }
    const int warps = 2;
    dim3 grid((s.N + warps - 1) / warps);
    if (D == 1) k_exch_energies<1><<<grid, warps * 32, 0, st>>>(s);
    else if (D == 2) k_exch_energies<2><<<grid, warps * 32, 0, st>>>(s);
    else k_exch_energies<3><<<grid, warps * 32, 0, st>>>(s);
    return 0;
}

// y of both directions for the banded solve and the multi-SM solve (and g
// for the multi-SM estimate before them), then the banded solve's store;
// publication flags for the multi-SM kernels.
size_t exchange_grid_doubles(const Sys& s) { return 2 * ((size_t)s.N + 1) + (band_store_floats(s) + 1) / 2; }
size_t exchange_grid_flags(const Sys& s) {
    return s.N >= kFlatEnergiesMinN ? 2 * (((size_t)s.N + 1 + 31) / 32) + 1 : 1;
}

// CTAs of kGridSolveThreads that are resident on the whole GPU at once, for
// kernel `which` (0 solve, 1 estimate) with up to 8 KB of dynamic shared
// memory; measured once per device.
static int grid_resident(int which) {
    static std::atomic<int> per_dev[2][64];  // 0 = not measured yet
    int dev = 0;
    cudaGetDevice(&dev);
    const bool known = dev >= 0 && dev < 64;
    int per = known ? per_dev[which][dev].load(std::memory_order_relaxed) - 1 : -1;
    if (per < 0) {
        int sms = 0, b = 0;
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        const void* k = which ? (const void*)k_exch_estimate_grid : (const void*)k_exch_solve_grid;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k, kGridSolveThreads, 8192) != cudaSuccess) b = 0;
        per = b * sms;
        if (known) per_dev[which][dev].store(per + 1, std::memory_order_relaxed);
    }
    return per;
}
// CTAs per direction of the multi-SM kernels and the 32-node blocks each owns at most.
static int grid_ctas(const Sys& s) { return std::min((s.N + 1 + 31) / 32, kGridSolveCtas); }
static size_t grid_owned(const Sys& s) { return (size_t)((s.N + 1 + 31) / 32 + grid_ctas(s) - 1) / grid_ctas(s); }

// The cooperative solve if every CTA can be resident; false otherwise.
static bool grid_solve(const Sys& s, int phase, double* ysol, unsigned* gflags, int banded, cudaStream_t st) {
    const int nct = grid_ctas(s);
    if (2 * nct > grid_resident(0)) return false;
    Sys sc = s;
    int ph = phase, n = nct, bd = banded;
    void* args[] = {&sc, &ph, &ysol, &gflags, &n, &bd};
    return cudaLaunchCooperativeKernel((void*)k_exch_solve_grid, dim3(2 * nct), dim3(kGridSolveThreads), args,
                                      sizeof(double) * (grid_owned(s) * 32 + 32), st) == cudaSuccess;
}
// The cooperative estimate likewise.
static bool grid_estimate(const Sys& s, int phase, double* ysol, unsigned* gflags, cudaStream_t st) {
    const int nct = grid_ctas(s);
    if (2 * nct > grid_resident(1)) return false;
    Sys sc = s;
    int ph = phase, n = nct;
    float* g = reinterpret_cast<float*>(ysol);
    void* args[] = {&sc, &ph, &g, &gflags, &n};
    return cudaLaunchCooperativeKernel((void*)k_exch_estimate_grid, dim3(2 * nct), dim3(kGridSolveThreads), args,
                                      sizeof(float) * 2 * grid_owned(s) * 32, st) == cudaSuccess;
}

// SMs the pair tiles leave free while this exchange runs beside them: its
// one-block passes (below the multi-SM solve's size) then run alone on an SM.
int exchange_reserved_sms(const Sys& s) { return s.N < kGridSolveMinN ? 2 : 0; }

// With `alone` the launch prefers a carveout of little more than its shared
// memory, so that its CTAs start on SMs without pair blocks (which run under the
// largest) and the dense solve reads the weights through a large L1: started
// under the pair blocks' carveout it keeps the small one to its end (dipoles of
// 711 particles, 7 beads, dense weights: 295 -> 271 us a step).  Not from 768
// particles, where the multi-SM solve waits for it (850, 32 beads: 243 -> 254).
static void launch_solve_band(const Sys& s, int phase, double* ysol, int standalone, size_t smem, bool alone,
                              cudaStream_t st) {
    cudaLaunchConfig_t c = {};
    c.gridDim = dim3(2);
    c.blockDim = dim3(kBandThreads);
    c.dynamicSmemBytes = smem;
    c.stream = st;
    cudaLaunchAttribute at = {};
    at.id = cudaLaunchAttributePreferredSharedMemoryCarveout;
    at.val.sharedMemCarveout = (unsigned)((smem + 4 * 1024) * 100 / (228 * 1024) + 1);
    c.attrs = &at;
    c.numAttrs = alone ? 1 : 0;
    cudaLaunchKernelEx(&c, k_exch_solve_band, s, phase, ysol, standalone);
}

int launch_exchange_recursions(const Sys& s, int exact, cudaStream_t st, double* ysol, unsigned* gflags,
                               int estimate_done) {
    exchange_carveouts();
    // With reserved SMs the one-block passes ask for 116 KB of shared memory,
    // whatever they use: more than an SM holding pair-tile blocks has left
    // and more than half an SM, so each lands alone on a reserved SM.
    const size_t least = s.reserve_sms ? 116 * 1024 : 0;
    const size_t esmem = std::max(sizeof(float) * 3 * (size_t)(s.N + 1), least);
    const size_t smem = std::max(sizeof(double) * (2 * (size_t)(s.N + 1) + 32), least);
    opt_in_smem((const void*)k_exch_estimate, esmem);
    opt_in_smem((const void*)k_exch_solve, smem);
    if (exact) {
        k_exch_solve<<<2, kWaveThreads, smem, st>>>(s, 1, 0, nullptr, 0);
        return 1;
    }
    // weights: rows or tiles by size; the retry's a small grid-stride launch
    const int tiles = tile_count(s.N);
    const dim3 wgrid((s.N + 255) / 256, s.N), rgrid(1, std::min(s.N, 256));
    // below the multi-SM solve's size a failed solve is retried inside
    // k_exch_solve (phase 0 only)
    const int inline_retry = s.N < kGridSolveMinN;
    // below the multi-SM solve's size the banded kernel is the whole pass 3
    const int standalone = inline_retry && ysol && banded_solve_fits(s);
    int n = 0;
    for (int phase = 0; phase < (inline_retry ? 1 : 2); ++phase) {
        if (!(phase == 0 && estimate_done)) {  // else the energy kernel ran it
            // across SMs from the flat energies' size, else on two blocks
            if (!(s.N >= kFlatEnergiesMinN && ysol && gflags && grid_estimate(s, phase, ysol, gflags, st)))
                k_exch_estimate<<<2, kWaveThreads, esmem, st>>>(s, phase);
            ++n;
        }
        if (!(phase == 0 && estimate_done)) {  // else the energy kernel formed them
            if (s.N < kTileWeightsMinN)
                k_exch_weights_rows<<<phase ? rgrid : wgrid, 256, 0, st>>>(s, phase);
            else
                k_exch_weights<<<phase ? std::min(tiles, 512) : tiles, kTileThreads, 0, st>>>(s, phase, tiles);
            ++n;
        }
        // the banded kernel (one CTA per direction): below the multi-SM
        // solve's size the whole pass 3, from it the banded case only
        int banded = 0;
        if (ysol && banded_solve_fits(s)) {
            const size_t bs = std::max(banded_solve_smem(s), least);
            opt_in_smem((const void*)k_exch_solve_band, bs);
            launch_solve_band(s, phase, ysol, standalone, bs, standalone && least, st);
            banded = 1;
            ++n;
        }
        if (standalone) continue;
        // from kGridSolveMinN the dense solve runs across SMs; below it (no
        // ysol) k_exch_solve solves on its own block
        const bool dense = ysol && !inline_retry && gflags && grid_solve(s, phase, ysol, gflags, banded, st);
        const bool pre = banded || dense;
        k_exch_solve<<<2, kWaveThreads, smem, st>>>(s, 0, phase, pre ? ysol : nullptr, inline_retry);
        n += dense ? 2 : 1;
    }
    return n;
}

static void exchange_rows(const Sys& s, int D, int accumulate, int adjoint, double vb_bar, cudaStream_t st) {
    exchange_carveouts();
    const int warps = 2;  // small blocks: the 2N rows spread over every SM
    dim3 grid((2 * s.N + warps - 1) / warps);
    if (D == 1) k_exch_forces<1><<<grid, warps * 32, 0, st>>>(s, accumulate, adjoint, vb_bar);
    else if (D == 2) k_exch_forces<2><<<grid, warps * 32, 0, st>>>(s, accumulate, adjoint, vb_bar);
    else k_exch_forces<3><<<grid, warps * 32, 0, st>>>(s, accumulate, adjoint, vb_bar);
}

void launch_exchange_forces_mode(const Sys& s, int D, int accumulate, cudaStream_t st) {
    exchange_rows(s, D, accumulate, 0, 0.0, st);
}

void launch_exchange_adjoint(const Sys& s, int D, double vb_bar, cudaStream_t st) {
    exchange_rows(s, D, 0, 1, vb_bar, st);
}

void launch_exchange_estimators(const Sys& s, cudaStream_t st) {
    const int rows = kEstimatorThreads / 32;
    k_exch_estimators<<<std::min((s.N + rows - 1) / rows, kEstimatorBlocks), kEstimatorThreads, 0, st>>>(s, s.P);
}

}  // namespace pimdb
