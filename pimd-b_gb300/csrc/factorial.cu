// Factorial bosonic exchange: the sum over all N! permutations of the
// exterior links between beads P and 1 (the reference's build with
// FACTORIAL_BOSONIC_ALGORITHM, CMakeLists.txt:49-54).
//
// Reference: FactorialBosonicExchange (src/bosonic_exchange/factorial_bosonic_exchange.cpp)
//   prepare :19-21, effectivePotential :91-114, springForceLastBead :121-172,
//   springForceFirstBead :179-230, primEstimator :259-293 -> k_factorial
//   getDistinctProbability :237-240, getLongestProbability :249-252 return 0
//
// For a given configuration this is a different potential from the
// Feldman-Hirshberg recursion (which keeps one representative cycle per set
// of exchanged particles); the two agree only after the interior beads are
// integrated out.
//
// The reference enumerates the permutations.  With d2[l][m] = |x_1[m] -
// x_P[l]|^2 (minimum image) and link energies e[l][m] = k/2 d2[l][m], a
// permutation's energy is the sum of its links', so its weight is a product
// of link factors A[l][m] = exp(-beta_ex e[l][m]) and the sum over
// permutations is the permanent of A.  It is summed over subsets instead:
//   F[c] = sum over the placements of the first |c| links on the targets c
//        = sum_{m in c} F[c \ m] A[|c|-1][m],
//   B[c] = the same for the links |c| .. N-1 on the targets outside c
//        = sum_{m not in c} A[|c|][m] B[c + m],
//   S = F[all],  M[l][m] = A[l][m] sum_{|c|=l, m not in c} F[c] B[c + m],
// M[l][m]/S being the probability that link l ends on m: N 2^(N-1) terms
// each instead of N!, all positive (no cancellation).  Then
//   f_P[l] = k (x_{P-1}[l] - x_P[l] + sum_m M[l][m]/S (x_1[m] - x_P[l]))
//   f_1[m] = k (x_2[m] - x_1[m] + sum_l M[l][m]/S (x_P[l] - x_1[m]))
// (each difference under the minimum image), V_B = -log(S/N!)/beta_ex and
// primEstimator = -(sum_{l,m} M[l][m]/S e[l][m])/P.
//
// Range.  beta_ex e[l][m] is taken relative to r_l + q_m, first r the rows'
// minima and q the columns' minima of the rest: every factor is then at most
// 1, and the shift joins V_B again.  Where even the best permutation falls
// below 1e-200 (links that compete for the same near targets, far from
// equilibrium), r and q become the potentials of the optimal assignment: the
// best permutation then has weight 1.
// (The reference's unshifted effectivePotential underflows to V_B = inf.)
//
// One block; F and B (64 KB at N = 12) in shared memory, one barrier per
// level.  Bound: the latency of 2 N levels and, from N = 11, one SM's FP64
// pipe (3 N 2^(N-1) multiply-adds).  Measured in a one-step run of N = 10,
// P = 8 from a new state: 485 us enumerating the 10! permutations on every SM
// (three kernels, 428 us of it), 125 us with this one.  Results are
// deterministic.
#include "forces_dev.cuh"
#include "kernels.h"

namespace pimdb {

namespace {

constexpr int kFactThreads = 1024;
constexpr double kFactSmallest = 1e-200;

__host__ __device__ constexpr double factorial_of(int n) {
    double r = 1.0;
    for (int i = 2; i <= n; ++i) r *= i;
    return r;
}

// Potentials r, q with r[l] + q[m] <= a[l][m], and equality on the cheapest
// permutation, by the whole block; `cost` (2^N doubles) is scratch.  The
// cheapest way to place the first |c| links on the targets c is found over
// subsets as F is, with minima for sums (dynamic programming over subsets:
// Held and Karp 1962), and the permutation sigma by walking it back.  With
// q[sigma(k)] = a[k][sigma(k)] - r[k] what remains are bounds on differences,
// r[l] - r[k] <= a[l][sigma(k)] - a[k][sigma(k)], which shortest paths satisfy
// (Bellman-Ford, N rounds: the cheapest permutation leaves no negative cycle).
__device__ __noinline__ void assignment_potentials(int N, const double* a, double* cost, int* sigma, double* r,
                                                   double* q) {
    const int tid = threadIdx.x, size = 1 << N;
    for (int n = 0; n <= N; ++n) {
        for (int c = tid; c < size; c += kFactThreads) {
            if (__popc(c) != n) continue;
            double least = n ? (double)INFINITY : 0.0;
            for (int w = c; w; w &= w - 1) {
                const int m = __ffs(w) - 1;
                least = fmin(least, cost[c ^ (1 << m)] + a[(n - 1) * N + m]);
            }
            cost[c] = least;
        }
        __syncthreads();
    }
    if (tid < 32) {
        if (tid == 0)
            for (int l = N - 1, c = size - 1; l >= 0; --l) {
                int take = __ffs(c) - 1;
                for (int w = c & (c - 1); w; w &= w - 1) {
                    const int m = __ffs(w) - 1;
                    if (cost[c ^ (1 << m)] + a[l * N + m] < cost[c ^ (1 << take)] + a[l * N + take]) take = m;
                }
                sigma[l] = take;
                c ^= 1 << take;
            }
        __syncwarp();
        const int l = tid < N ? tid : 0;
        double d = 0.0;
        for (int round = 0; round < N; ++round) {
            if (tid < N) r[tid] = d;
            __syncwarp();
            for (int k = 0; k < N; ++k) d = fmin(d, r[k] + (a[l * N + sigma[k]] - a[k * N + sigma[k]]));
            __syncwarp();
        }
        if (tid < N) {
            r[tid] = d;
            q[sigma[tid]] = a[tid * N + sigma[tid]] - d;
        }
    }
    __syncthreads();
}

// The sum over permutations, the scalars and the exterior spring forces of
// beads 1 and P into fx (and added into f with `accumulate`).  One block.
template <int D>
__global__ void __launch_bounds__(kFactThreads) k_factorial(Sys s, int accumulate) {
    extern __shared__ double sub[];  // F, B: 2^N each
    __shared__ double d2[kFactMaxN * kFactMaxN];
    __shared__ double ar[kFactMaxN * kFactMaxN];  // beta_ex e
    __shared__ double A[kFactMaxN * kFactMaxN];
    __shared__ double M[kFactMaxN * kFactMaxN];
    __shared__ double r[kFactMaxN], q[kFactMaxN];
    __shared__ int sigma[kFactMaxN];
    const int tid = threadIdx.x, N = s.N, NN = N * N, size = 1 << N;
    const int lane = tid & 31, warp = tid >> 5, nw = kFactThreads / 32;
    double* F = sub;
    double* B = sub + size;
    const double ka = 0.5 * s.kappa * s.beta_ex;
    if (tid < NN) {
        const int l = tid / N, m = tid - l * N;
        double acc = 0.0;
#pragma unroll
        for (int a = 0; a < D; ++a) {
            double d = s.x[idx<D>(s, 0, a, m)] - s.x[idx<D>(s, s.P - 1, a, l)];
            if (s.pbc) d = min_image(d, s.L, s.invL);
            acc += d * d;
        }
        d2[tid] = acc;
        ar[tid] = ka * acc;
    }
    __syncthreads();
    if (tid < N) {
        double t = ar[tid * N];
        for (int m = 1; m < N; ++m) t = fmin(t, ar[tid * N + m]);
        r[tid] = t;
    }
    __syncthreads();
    if (tid < N) {
        double t = ar[tid] - r[0];
        for (int l = 1; l < N; ++l) t = fmin(t, ar[l * N + tid] - r[l]);
        q[tid] = t;
    }
    __syncthreads();
    for (int attempt = 0; attempt < 2; ++attempt) {
        if (tid < NN) {
            const int l = tid / N, m = tid - l * N;
            A[tid] = exp(-((ar[tid] - r[l]) - q[m]));
        }
        if (tid == 0) {
            F[0] = 1.0;
            B[size - 1] = 1.0;
        }
        __syncthreads();
        // level by level: the lower half of the block takes F upwards, the
        // upper half B downwards (small N: half a block is plenty)
        constexpr int kHalf = kFactThreads / 2;
        const bool up = tid < kHalf;
        for (int lev = 1; lev <= N; ++lev) {
            const int n = up ? lev : N - lev;  // the subsets' size
            const double* row = A + (up ? n - 1 : n) * N;
            for (int c = tid & (kHalf - 1); c < size; c += kHalf) {
                if (__popc(c) != n) continue;
                double t0 = 0.0, t1 = 0.0;
                for (unsigned w = up ? c : ~c & (size - 1); w;) {
                    const int m = __ffs(w) - 1;
                    w &= w - 1u;
                    const int o = c ^ (1 << m);
                    t0 = fma(up ? F[o] : B[o], row[m], t0);
                    if (w) {
                        const int m1 = __ffs(w) - 1;
                        w &= w - 1u;
                        const int o1 = c ^ (1 << m1);
                        t1 = fma(up ? F[o1] : B[o1], row[m1], t1);
                    }
                }
                if (up) F[c] = t0 + t1;
                else B[c] = t0 + t1;
            }
            __syncthreads();
        }
        const double S = F[size - 1];
        if (S >= kFactSmallest || !isfinite(S) || attempt) break;  // the whole block alike
        __syncthreads();
        assignment_potentials(N, ar, F, sigma, r, q);
    }
    const double S = F[size - 1], invS = 1.0 / S;
    // M[l][m]: one warp per entry over the subsets without m
    for (int e = warp; e < NN; e += nw) {
        const int l = e / N, m = e - l * N, low = (1 << m) - 1;
        double t = 0.0;
        for (int k = lane; k < size >> 1; k += 32) {
            if (__popc(k) != l) continue;
            const int c = ((k & ~low) << 1) | (k & low);
            t = fma(F[c], B[c | (1 << m)], t);
        }
        t = warp_sum(t);
        if (lane == 0) M[e] = t * A[e] * invS;
    }
    __syncthreads();
    if (warp == 0) {
        double pe = 0.0, shift = 0.0;
        for (int e = lane; e < NN; e += 32) pe = fma(M[e], d2[e], pe);
        if (lane < N) shift = r[lane] + q[lane];
        pe = warp_sum(pe);
        shift = warp_sum(shift);
        if (lane == 0) {
            if (!(S > 0.0) || !isfinite(S) || !isfinite(pe) || !isfinite(shift)) atomicOr(s.err, ERRB_NONFINITE_VB);
            s.scal[0] = (shift - log(S / factorial_of(N))) / s.beta_ex;
            s.scal[1] = -(0.5 * s.kappa * pe) / s.P;
            s.scal[2] = 0.0;
            s.scal[3] = 0.0;
        }
    }
    const int first = 0, last = s.P - 1;
    // one thread per particle, bead and axis (the upper warps: warp 0 is busy)
    for (int t = kFactThreads - 1 - tid; t < 2 * N * D; t += kFactThreads) {
        const int w = t / D, a = t - w * D;
        const bool is_last = w < N;
        const int l = is_last ? w : w - N;
        const int bead = is_last ? last : first;
        const int other = is_last ? first : last;
        const int nb = is_last ? (s.P - 2 + s.P) % s.P : 1 % s.P;
        const int side = is_last ? 1 : 0;
        const double xl = s.x[idx<D>(s, bead, a, l)];
        double sum = 0.0;
        for (int k = 0; k < N; ++k) {
            double d = s.x[idx<D>(s, other, a, k)] - xl;
            if (s.pbc) d = min_image(d, s.L, s.invL);
            sum += (is_last ? M[l * N + k] : M[k * N + l]) * d;
        }
        double di = s.x[idx<D>(s, nb, a, l)] - xl;
        if (s.pbc) di = min_image(di, s.L, s.invL);
        const double fs = (sum + di) * s.kappa;
        s.fx[((size_t)side * D + a) * s.ld + l] = fs;
        if (accumulate) {
            const size_t o = idx<D>(s, bead, a, l);
            s.f[o] = fs + s.f[o];
        }
    }
}

template <int D>
void factorial_launch(const Sys& s, int accumulate, cudaStream_t st) {
    const size_t smem = 2 * sizeof(double) * ((size_t)1 << s.N);
    if (smem + 8 * 1024 > 48 * 1024)  // the static arrays (5 KB) count too
        cudaFuncSetAttribute(k_factorial<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    k_factorial<D><<<1, kFactThreads, smem, st>>>(s, accumulate);
}

}  // namespace

void launch_factorial(const Sys& s, int D, int accumulate, cudaStream_t st) {
    if (D == 1) factorial_launch<1>(s, accumulate, st);
    else if (D == 2) factorial_launch<2>(s, accumulate, st);
    else factorial_launch<3>(s, accumulate, st);
}

}  // namespace pimdb
