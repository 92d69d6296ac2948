// The lowest eigenpairs of a large sparse symmetric positive semi-definite
// matrix on the device, by Chebyshev-filtered subspace iteration in float64.
//
// Used for the port-mode problems of large port planes, where a dense
// eigensolve (modes.cu) is out of reach: the TE modes of a hollow guide as
// the face form L = B B^T, B = W^1/2 C M^-1/2 (C the face circulations of
// the plane's free edges, W = 1/M_mu of the normal-H faces, M the edge
// epsilon-masses), whose nonzero spectrum is that of the edge problem
// K v = lambda M v the reference solves with shift-invert ARPACK
// (src/magnelio/ports/_modal/numerical_2d.py:497-544) and whose null space
// is one known vector per connected face region; and the TM problem on the
// plane's normal edges (curl_curl_2d.py:127-218), positive definite.
//
// One iteration: the block X (n x k, k > n_modes) is passed through the
// Chebyshev polynomial of degree m <= 100 that is bounded by 1 on [a, b]
// (b an upper bound of the spectrum, a the largest Ritz value of the
// block) and grows fast below a (the scaled three-term recurrence, one
// fused SpMM per degree; m capped so that the gain at the lowest Ritz
// value stays near 1e8); the caller's null vectors are projected out; the block is
// orthonormalised by classical Gram-Schmidt with reorthogonalisation; the
// Rayleigh-Ritz step (H = X^T L X, a k x k Jacobi eigensolve on the host)
// rotates it onto the Ritz vectors; the residuals ||L x_j - theta_j x_j||
// decide convergence.  Every loop is bounded; the routine reports the
// iterations used and fails if the residuals do not reach the tolerance.
//
// A port plane's block (a few thousand rows, seven columns) is far too small
// to fill the chip: the time is launches and host round trips.  So a filter
// (up to 100 degrees) and the orthonormalisation of a block are one
// cooperative launch each, their CTAs meeting at bounded grid barriers: on a
// 104 x 46 plane with three modes the solve took 8.5 ms with a launch per
// degree and some eight launches and two host reads per column, and 4.8 ms so
// (7 iterations; 209 x 93: 24 and 12.8 ms).  A call's allocations and frees come
// on top and vary with what else the process holds (5 to 9 ms in all).
#include "fitb_common.cuh"

#include <algorithm>
#include <cmath>
#include <vector>

namespace fitb {

namespace {

constexpr int kT = 256;

int grid_for(long long work) {
    return (int)std::max<long long>(1, std::min<long long>((work + kT - 1) / kT, 148LL * 16));
}

__device__ double block_reduce(double x, double* sh) {
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = x;
    __syncthreads();
    double r = 0.0;
    if (threadIdx.x == 0)
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) r += sh[w];
    return r;
}

// Barrier of all CTAs of a cooperative launch: `bar` counts arrivals (zeroed
// before the launch), `round` is the caller's count of barriers so far.  The
// wait is bounded; an expired one sets *err to 1 and every later barrier falls
// through.  (Another *err is no reason to leave: it may be set by a CTA that is
// already past the barrier that this one still leaves.)
constexpr unsigned kBarrierLimit = 1u << 24;
__device__ __forceinline__ void grid_barrier(unsigned* bar, unsigned& round, int* err) {
    __syncthreads();
    if (threadIdx.x == 0) {
        const unsigned target = ++round * gridDim.x * gridDim.y;
        __threadfence();
        atomicAdd(bar, 1u);
        unsigned v, tries = 0;
        do {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(bar) : "memory");
        } while ((int)(v - target) < 0 && ++tries < kBarrierLimit && *(volatile int*)err != 1);
        if ((int)(v - target) < 0) atomicExch(err, 1);
        __threadfence();
    }
    __syncthreads();
}

// Yn = alpha (L Y) + beta Y + gamma X, blocks column-major (column j at j n)
__global__ void k_cheb(long long n, int k, const long long* rp, const long long* col, const double* val,
                       const double* Y, const double* X, double* Yn, double alpha, double beta, double gamma) {
    const long long total = n * k;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < total;
         t += (long long)gridDim.x * blockDim.x) {
        const long long j = t / n, i = t - j * n;
        const double* y = Y + j * n;
        double acc = 0.0;
        for (long long q = rp[i]; q < rp[i + 1]; ++q) acc += val[q] * y[col[q]];
        double r = alpha * acc + beta * y[i];
        if (gamma != 0.0) r += gamma * X[t];
        Yn[t] = r;
    }
}

// a reproducible start block: a hash of (row, column, seed) in [-1, 1)
__device__ __forceinline__ double random_entry(long long r, long long c, unsigned seed) {
    unsigned long long h = (unsigned long long)r * 0x9E3779B97F4A7C15ull ^
                           ((unsigned long long)(c + 1) * 0xBF58476D1CE4E5B9ull) ^ ((unsigned long long)seed << 32);
    h ^= h >> 31;
    h *= 0x94D049BB133111EBull;
    h ^= h >> 29;
    return (double)(h >> 11) * (2.0 / 9007199254740992.0) - 1.0;
}

// The whole filter: degree d (from 1) of the recurrence with the factors
// f[3 (d-1) ..], from P0 (the block) through P1, P2 in rotation; the last
// degree's block is P[m % 3].  Other CTAs' rows change between degrees, so
// they are read past the L1.
struct ChebPlan {
    double f[300];
    double* P[3];
    int m;
};
constexpr int kTF = 512;  // few CTAs, so that few meet at the barriers; column blockIdx.y
__global__ void __launch_bounds__(kTF) k_filter(long long n, const long long* __restrict__ rp,
                                               const long long* __restrict__ col, const double* __restrict__ val,
                                               const __grid_constant__ ChebPlan p, unsigned* bar, int* err) {
    unsigned round = 0;
    const long long c0 = blockIdx.y * n;
    for (int d = 1; d <= p.m; ++d) {
        const double alpha = p.f[3 * d - 3], beta = p.f[3 * d - 2], gamma = p.f[3 * d - 1];
        const double* y = p.P[(d - 1) % 3] + c0;
        const double* x = p.P[(d + 1) % 3] + c0;  // the degree before y's
        double* yn = p.P[d % 3] + c0;
        for (long long i = blockIdx.x * (long long)kTF + threadIdx.x; i < n; i += (long long)gridDim.x * kTF) {
            const double prev = d > 1 ? x[i] : 0.0;
            double acc = 0.0;
            for (long long q = rp[i]; q < rp[i + 1]; ++q) acc += val[q] * __ldcg(y + col[q]);
            double r = alpha * acc + beta * __ldcg(y + i);
            if (d > 1) r += gamma * prev;
            yn[i] = r;
        }
        if (d < p.m) grid_barrier(bar, round, err);
    }
}

// The columns of X orthonormal to the nz vectors Z and to one another:
// classical Gram-Schmidt twice per column, a column that lost its rank
// started afresh (up to four times, then *err = 2).  part: one row of partial
// sums per CTA; they are added in CTA order, so the result does not depend on
// timing.
constexpr int kPart = 64;        // partial sums per CTA: nz + k + 1 of them used
constexpr int kOrthoCtas = 128;  // CTAs at most
__global__ void __launch_bounds__(kT) k_ortho(long long n, double* X, int k, const double* Z, int nz, double* part,
                                              unsigned* bar, int* err) {
    __shared__ double sh[32], coef[kPart];
    unsigned round = 0, flip = 0;
    const long long r0 = blockIdx.x * (long long)blockDim.x + threadIdx.x, stride = (long long)gridDim.x * blockDim.x;
    // coef[q] = (q < nz ? Z_q : X_(q - nz)) . x for q < nc, and x . x at nc
    // (two rows of partial sums in turn: one is written while a slower CTA
    // still reads the other)
    auto dots = [&](const double* x, int nc, bool cross) {
        double* pt = part + (size_t)(flip ^= 1u) * kOrthoCtas * kPart;
        for (int q = cross ? 0 : nc; q <= nc; ++q) {
            const double* a = q == nc ? x : (q < nz ? Z + (long long)q * n : X + (long long)(q - nz) * n);
            double s = 0.0;
            for (long long r = r0; r < n; r += stride) s += a[r] * x[r];
            s = block_reduce(s, sh);
            if (threadIdx.x == 0) pt[blockIdx.x * kPart + q] = s;
            __syncthreads();
        }
        grid_barrier(bar, round, err);
        for (int q = (cross ? 0 : nc) + (int)threadIdx.x; q <= nc; q += blockDim.x) {
            double s = 0.0;
            for (unsigned c = 0; c < gridDim.x; ++c) s += __ldcg(pt + c * kPart + q);
            coef[q] = s;
        }
        __syncthreads();
    };
    for (int c = 0; c < k; ++c) {
        double* x = X + (long long)c * n;
        const int nc = nz + c;
        bool done = false;
        for (int attempt = 0; attempt < 4 && !done; ++attempt) {
            double before = 0.0;
            for (int pass = 0; pass < 2; ++pass) {
                dots(x, nc, true);
                if (pass == 0) before = coef[nc];
                for (long long r = r0; r < n; r += stride) {
                    double s = 0.0;
                    for (int q = 0; q < nc; ++q)
                        s += coef[q] * (q < nz ? Z[(long long)q * n + r] : X[(long long)(q - nz) * n + r]);
                    x[r] -= s;
                }
            }
            dots(x, nc, false);
            const double after = coef[nc];
            done = after > 1e-20 * before && after > 0.0;
            const double f = done ? 1.0 / sqrt(after) : 0.0;
            for (long long r = r0; r < n; r += stride)
                x[r] = done ? x[r] * f : random_entry(r, c, 7919u * (attempt + 1) + 13u);
        }
        if (!done) {
            if (r0 == 0) atomicExch(err, 2);
            return;  // every CTA: `after` is the same in all of them
        }
    }
}

// out[i * nb + j] = A_i . B_j for i < na, j < nb (one block per pair)
__global__ void __launch_bounds__(kT) k_gram(long long n, const double* A, int na, const double* B, int nb,
                                             double* out) {
    __shared__ double sh[32];
    const int i = blockIdx.x / nb, j = blockIdx.x - (blockIdx.x / nb) * nb;
    if (i >= na) return;
    const double* a = A + (long long)i * n;
    const double* b = B + (long long)j * n;
    double s = 0.0;
    for (long long r = threadIdx.x; r < n; r += blockDim.x) s += a[r] * b[r];
    s = block_reduce(s, sh);
    if (threadIdx.x == 0) out[i * nb + j] = s;
}

// Out_j = sum_i In_i R[i * k + j]
__global__ void k_rotate(long long n, int k, const double* In, const double* R, double* Out) {
    const long long total = n * k;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < total;
         t += (long long)gridDim.x * blockDim.x) {
        const long long j = t / n, r = t - j * n;
        double s = 0.0;
        for (int i = 0; i < k; ++i) s += In[(long long)i * n + r] * R[i * k + j];
        Out[t] = s;
    }
}

// out[j] = || W_j - theta_j X_j ||^2 (one block per column)
__global__ void __launch_bounds__(kT) k_residual(long long n, const double* W, const double* X, const double* theta,
                                                 double* out) {
    __shared__ double sh[32];
    const long long j = blockIdx.x;
    const double th = theta[j];
    double s = 0.0;
    for (long long r = threadIdx.x; r < n; r += blockDim.x) {
        const double d = W[j * n + r] - th * X[j * n + r];
        s += d * d;
    }
    s = block_reduce(s, sh);
    if (threadIdx.x == 0) out[j] = s;
}

__global__ void k_random(long long n, int c0, int nc, unsigned seed, double* X) {
    const long long total = n * nc;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < total;
         t += (long long)gridDim.x * blockDim.x) {
        const long long c = t / n + c0, r = t - (t / n) * n;
        X[c * n + r] = random_entry(r, c, seed);
    }
}

// symmetric k x k eigen-decomposition by cyclic Jacobi sweeps (bounded):
// values ascending, vectors as the columns of V (row-major k x k)
void jacobi_eigen(int k, std::vector<double> A, std::vector<double>& w, std::vector<double>& V) {
    V.assign((size_t)k * k, 0.0);
    for (int i = 0; i < k; ++i) V[i * k + i] = 1.0;
    for (int sweep = 0; sweep < 100; ++sweep) {
        double off = 0.0, diag = 0.0;
        for (int i = 0; i < k; ++i) {
            diag += A[i * k + i] * A[i * k + i];
            for (int j = i + 1; j < k; ++j) off += A[i * k + j] * A[i * k + j];
        }
        if (off <= 1e-34 * diag || off == 0.0) break;
        for (int p = 0; p < k; ++p)
            for (int q = p + 1; q < k; ++q) {
                const double apq = A[p * k + q];
                if (apq == 0.0) continue;
                const double theta = (A[q * k + q] - A[p * k + p]) / (2.0 * apq);
                const double t = (theta >= 0 ? 1.0 : -1.0) / (std::fabs(theta) + std::sqrt(theta * theta + 1.0));
                const double c = 1.0 / std::sqrt(t * t + 1.0), s = t * c;
                for (int r = 0; r < k; ++r) {
                    const double arp = A[r * k + p], arq = A[r * k + q];
                    A[r * k + p] = c * arp - s * arq;
                    A[r * k + q] = s * arp + c * arq;
                }
                for (int r = 0; r < k; ++r) {
                    const double apr = A[p * k + r], aqr = A[q * k + r];
                    A[p * k + r] = c * apr - s * aqr;
                    A[q * k + r] = s * apr + c * aqr;
                }
                for (int r = 0; r < k; ++r) {
                    const double vrp = V[r * k + p], vrq = V[r * k + q];
                    V[r * k + p] = c * vrp - s * vrq;
                    V[r * k + q] = s * vrp + c * vrq;
                }
            }
    }
    std::vector<int> ord(k);
    for (int i = 0; i < k; ++i) ord[i] = i;
    std::sort(ord.begin(), ord.end(), [&](int a, int b) { return A[a * k + a] < A[b * k + b]; });
    std::vector<double> Vs((size_t)k * k);
    w.resize(k);
    for (int j = 0; j < k; ++j) {
        w[j] = A[ord[j] * k + ord[j]];
        for (int r = 0; r < k; ++r) Vs[r * k + j] = V[r * k + ord[j]];
    }
    V.swap(Vs);
}

}  // namespace

int sparse_lowest_eigs(long long n, const long long* rp, const long long* col, const double* val, int n_null,
                       const double* Z, int n_modes, double tol, double b, double* lam_out, double* vec_out,
                       double* res_out, int* iters_out, cudaStream_t s) {
    if (n < 2 || n_modes < 1 || n_modes > 16 || n_null < 0 || n_null > 8) return -1;
    const int k = (int)std::min<long long>(n_modes + std::max(4, n_modes), n - n_null);
    if (k < n_modes || !(b > 0.0)) return -1;
    const size_t blk = (size_t)n * k;
    // five allocations of a few hundred KB rather than one: the driver serves
    // those from chunks it holds, while one of more than a MB is mapped and
    // unmapped on every call (measured: 5.4 ms a call against 8.6)
    double *X = nullptr, *Y = nullptr, *Yn = nullptr, *W = nullptr, *sm = nullptr;
    auto release = [&]() { cudaFree(X), cudaFree(Y), cudaFree(Yn), cudaFree(W), cudaFree(sm); };
    if (cudaMalloc(&X, blk * 8) || cudaMalloc(&Y, blk * 8) || cudaMalloc(&Yn, blk * 8) || cudaMalloc(&W, blk * 8) ||
        cudaMalloc(&sm, (4096 + 2 * (size_t)kOrthoCtas * kPart) * 8)) {
        release();
        return -2;
    }
    double* H = sm + 64;        // k x k
    double* R = sm + 64 + 1024; // k x k
    double* th = sm + 64 + 2048;
    double* rs = sm + 64 + 2048 + 64;
    const int g_blk = grid_for((long long)blk);
    auto host_read = [&](const double* d, double* h, int cnt) {
        cudaMemcpyAsync(h, d, cnt * sizeof(double), cudaMemcpyDeviceToHost, s);
        return cudaStreamSynchronize(s) == cudaSuccess;
    };
    // cooperative launches: as many CTAs as the rows need and the chip holds
    int dev = 0, sms = 148, occ_f = 1;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ_f, k_filter, kTF, 0);
    const dim3 g_f((unsigned)std::max<long long>(1, std::min<long long>((n + kTF - 1) / kTF, (long long)sms * occ_f / k)),
                   (unsigned)k);
    const int g_o = (int)std::max<long long>(1, std::min<long long>((n + kT - 1) / kT, std::min(sms, kOrthoCtas)));
    unsigned* bar = reinterpret_cast<unsigned*>(sm + 64 + 2048 + 256);
    int* err = reinterpret_cast<int*>(bar + 1);
    double* part = sm + 4096;
    auto coop = [&](const void* f, dim3 grid, int threads, void** args) {
        if (cudaMemsetAsync(bar, 0, 2 * sizeof(unsigned), s) != cudaSuccess) return -2;
        return cudaLaunchCooperativeKernel(f, grid, dim3(threads), args, 0, s) == cudaSuccess ? 0 : -2;
    };
    // every column of X orthonormal to the null vectors and to the ones before
    // it; the outcome is read with the next host read
    auto ortho = [&]() -> int {
        long long nn = n;
        int kk = k, nz = n_null;
        const double* z = Z;
        double* x = X;
        void* args[] = {&nn, &x, &kk, &z, &nz, &part, &bar, &err};
        return coop((const void*)k_ortho, dim3(g_o), kT, args);
    };
    auto outcome = [&](int e) { return e == 2 ? -5 : (e ? -2 : 0); };
    std::vector<double> hH((size_t)k * k), w, V, hres(k);
    double a = 0.0, a0 = 0.0, best = 1e300;
    int since_best = 0, it = 0, rc = -4;
    auto rayleigh_ritz = [&]() -> int {
        k_cheb<<<g_blk, kT, 0, s>>>(n, k, rp, col, val, X, X, W, 1.0, 0.0, 0.0);
        k_gram<<<k * k, kT, 0, s>>>(n, X, k, W, k, H);
        int e = 0;
        cudaMemcpyAsync(&e, err, sizeof(int), cudaMemcpyDeviceToHost, s);
        if (!host_read(H, hH.data(), k * k)) return -2;
        if (e) return outcome(e);
        for (int i = 0; i < k; ++i)
            for (int j = i + 1; j < k; ++j) hH[i * k + j] = hH[j * k + i] = 0.5 * (hH[i * k + j] + hH[j * k + i]);
        jacobi_eigen(k, hH, w, V);
        cudaMemcpyAsync(R, V.data(), (size_t)k * k * sizeof(double), cudaMemcpyHostToDevice, s);
        cudaMemcpyAsync(th, w.data(), k * sizeof(double), cudaMemcpyHostToDevice, s);
        k_rotate<<<g_blk, kT, 0, s>>>(n, k, X, R, Y);
        k_rotate<<<g_blk, kT, 0, s>>>(n, k, W, R, Yn);
        std::swap(X, Y);
        std::swap(W, Yn);
        k_residual<<<k, kT, 0, s>>>(n, W, X, th, rs);
        if (!host_read(rs, hres.data(), k)) return -2;
        return 0;
    };
    k_random<<<g_blk, kT, 0, s>>>(n, 0, k, 1u, X);
    int e0 = ortho();
    if (e0 == 0) e0 = rayleigh_ritz();
    if (e0) {
        release();
        return e0;
    }
    const int degree = 100, max_iter = 400;
    for (it = 1; it <= max_iter; ++it) {
        a = w[k - 1];
        a0 = std::min(w[0], 0.5 * a);
        if (!(a < b)) a = 0.5 * b;
        // Chebyshev filter of degree `degree` on [a, b], scaled to 1 at a0
        const double e = 0.5 * (b - a), c = 0.5 * (b + a);
        double sigma = e / (a0 - c);
        const double tau = 2.0 / sigma;
        // degree: at most `degree`, and low enough that the filter's gain at
        // the lowest Ritz value over its bound on [a, b] stays near 1e8 (a
        // higher gain would fold the whole block onto one vector)
        const double x0 = (a + b - 2.0 * a0) / (b - a);
        const int m = (int)std::min<double>(degree, std::max(1.0, 19.0 / std::acosh(std::max(x0, 1.0 + 1e-12))));
        ChebPlan plan;
        plan.m = m;
        plan.P[0] = X;
        plan.P[1] = Y;
        plan.P[2] = Yn;
        plan.f[0] = sigma / e;
        plan.f[1] = -c * sigma / e;
        plan.f[2] = 0.0;
        for (int d = 2; d <= m; ++d) {
            const double s2 = 1.0 / (tau - sigma);
            plan.f[3 * d - 3] = 2.0 * s2 / e;
            plan.f[3 * d - 2] = -2.0 * s2 * c / e;
            plan.f[3 * d - 1] = -sigma * s2;
            sigma = s2;
        }
        long long nn = n;
        void* args[] = {&nn, &rp, &col, &val, &plan, &bar, &err};
        int er = coop((const void*)k_filter, g_f, kTF, args);
        // the filtered block to X
        X = plan.P[m % 3];
        Y = plan.P[(m + 1) % 3];
        Yn = plan.P[(m + 2) % 3];
        int ferr = 0;
        if (er == 0 && cudaMemcpyAsync(&ferr, err, sizeof(int), cudaMemcpyDeviceToHost, s) != cudaSuccess) er = -2;
        if (er == 0) er = ortho();
        if (er == 0) er = rayleigh_ritz();
        if (er == 0) er = outcome(ferr);
        if (er) {
            release();
            return er;
        }
        double worst = 0.0;
        for (int j = 0; j < n_modes; ++j) worst = std::max(worst, std::sqrt(std::max(hres[j], 0.0)) / b);
        if (worst <= tol) {
            rc = 0;
            break;
        }
        // residuals stuck at the rounding floor: accept once below 1e-12 b
        if (worst < 0.5 * best) {
            best = worst;
            since_best = 0;
        } else if (++since_best >= 20 && worst <= 1e-12) {
            rc = 0;
            break;
        }
    }
    double worst = 0.0;
    for (int j = 0; j < n_modes; ++j) worst = std::max(worst, std::sqrt(std::max(hres[j], 0.0)) / b);
    if (res_out) *res_out = worst;
    if (iters_out) *iters_out = it;
    if (rc == 0) {
        for (int j = 0; j < n_modes; ++j) lam_out[j] = w[j];
        cudaMemcpyAsync(vec_out, X, (size_t)n_modes * n * sizeof(double), cudaMemcpyDeviceToHost, s);
        if (cudaStreamSynchronize(s) != cudaSuccess) rc = -2;
    }
    if (cudaGetLastError() != cudaSuccess) rc = -2;
    release();
    return rc;
}

}  // namespace fitb
