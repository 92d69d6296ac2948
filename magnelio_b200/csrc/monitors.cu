// Running-DFT field monitors, blocked in time.
//
// Reference: MonitorFieldFrequency.record
// (src/magnelio/monitors/field_frequency.py:249-294) interpolates the
// staggered states to cell centres (src/magnelio/monitors/base.py:51-168)
// and adds bins[f] += exp(j w_f t) dt_w * data (src/magnelio/monitors/_dft.py
// :37-52) every recorded step, with t = n dt for E and (n + 1/2) dt for H.
//
// Here each recorded step only stages the interpolated float32 samples and
// the float64-evaluated phasors exp(j w t) dt_w of that step into a block of
// K slots.  On the step that fills the block, the thread that staged a cell's
// samples forms sum_s w_s[f] x_s for every bin of that cell in registers and
// adds it once to the bins (optionally Kahan-compensated): the complex bins
// are read and written once per K recorded steps instead of once per step.
// All monitors share this one launch per step (k_dft_step).
#include "fitb_common.cuh"

namespace fitb {

namespace {

constexpr int kMaxK = 32;
constexpr int kThreads = 256;

__device__ __forceinline__ long long recorded_upto(long long x, int stride) {
    // Number of steps n' in [0, x] with n' % stride == 0 (0 for x < 0).
    return (x < 0) ? 0 : x / stride + 1;
}

template <typename T>
__device__ __forceinline__ double interp_sample(const T* E, const T* H, long long vol, const Geom& g,
                                                const DftDev& d, int c, int i, int j, int k) {
    const long long o = pidx(g, i, j, k);
    const double* dx = d.inv;
    const double* dy = d.inv + d.inv_ld;
    const double* dz = d.inv + 2 * d.inv_ld;
    const double* dxa = d.dual;
    const double* dya = d.dual + d.inv_ld;
    const double* dza = d.dual + 2 * d.inv_ld;
    const long long si = g.si, sj = g.sj;
    switch (c) {
        case 0: {
            const T* A = E;
            T s = ((A[o] + A[o + sj]) + A[o + 1]) + A[o + sj + 1];
            return (double)(T(0.25) * s) / dx[i];
        }
        case 1: {
            const T* A = E + vol;
            T s = ((A[o] + A[o + si]) + A[o + 1]) + A[o + si + 1];
            return (double)(T(0.25) * s) / dy[j];
        }
        case 2: {
            const T* A = E + 2 * vol;
            T s = ((A[o] + A[o + si]) + A[o + sj]) + A[o + si + sj];
            return (double)(T(0.25) * s) / dz[k];
        }
        case 3: {
            const T* A = H;
            return 0.5 * ((double)A[o] / dxa[i] + (double)A[o + si] / dxa[i + 1]);
        }
        case 4: {
            const T* A = H + vol;
            return 0.5 * ((double)A[o] / dya[j] + (double)A[o + sj] / dya[j + 1]);
        }
        default: {
            const T* A = H + 2 * vol;
            return 0.5 * ((double)A[o] / dza[k] + (double)A[o + 1] / dza[k + 1]);
        }
    }
}

__device__ __forceinline__ int monitor_of_block(const DftDev* devs, int nmon) {
    int m = 0;
    while (m + 1 < nmon && (int)blockIdx.x >= devs[m + 1].sblk0) ++m;
    return m;
}

// Adds kc staged samples x[s * xs] (s < n_st) and, at s = kc - 1, `last` to
// the bins of one cell-component: bins bi + f * ncell, phasors sw.
__device__ __forceinline__ void flush_cell(const DftDev& d, int kc, int tsel, const float* x, long long xs, int n_st,
                                           float last, long long bi, const float2* sw) {
    float v[kMaxK];
#pragma unroll
    for (int s = 0; s < kMaxK; ++s) v[s] = s < n_st ? x[s * xs] : (s == kc - 1 ? last : 0.0f);
    for (int f = 0; f < d.nf; ++f, bi += d.ncell) {
        float re = 0.0f, im = 0.0f;
#pragma unroll
        for (int s = 0; s < kMaxK; ++s) {
            if (s < kc) {
                const float2 w = sw[(s * 2 + tsel) * d.nf + f];
                re = fmaf(w.x, v[s], re);
                im = fmaf(w.y, v[s], im);
            }
        }
        float2 acc = d.bins[bi];
        if (d.kahan) {
            float2 cm = d.cmp[bi];
            const float yr = re - cm.x, yi = im - cm.y;
            const float tr = acc.x + yr, ti = acc.y + yi;
            cm.x = (tr - acc.x) - yr;
            cm.y = (ti - acc.y) - yi;
            acc.x = tr;
            acc.y = ti;
            d.cmp[bi] = cm;
        } else {
            acc.x += re;
            acc.y += im;
        }
        d.bins[bi] = acc;
    }
}

// One step of every monitor.  The step counter is *step - done: done = 1 when
// an earlier kernel of the step has advanced it; otherwise the last CTA of
// this launch does, through `ticket`.  Staging and flushing were two launches
// before, the second one empty on K - 1 of K steps: on a 97 x 104 x 89 mesh
// with three planes of 16 frequencies the two cost 13 us per step.  The
// launch is short, so its chain counts: up to kDftPack descriptors travel as
// kernel arguments (else a block's first loads are a descriptor from HBM or
// L2, one after the other per monitor), and the slot arithmetic is 32-bit
// while the step count is.
template <typename T, bool PACK>
__global__ void __launch_bounds__(kThreads, 3)
    k_dft_step(const T* __restrict__ e, const T* __restrict__ h, long long e_block, long long h_block, Geom g, int B,
               const __grid_constant__ DftPack pack, const DftDev* __restrict__ devs_dev, int nmon, long long* step,
               int done, unsigned* ticket) {
    extern __shared__ float2 sw[];
    const DftDev* devs = PACK ? pack.d : devs_dev;
    const DftDev& d = devs[monitor_of_block(devs, nmon)];
    const int lb = blockIdx.x - d.sblk0;
    const long long n = *step - done;
    const long long base = *d.base;
    const bool narrow = n < 0x7fffffffLL;
    if (narrow ? (unsigned)n % (unsigned)d.stride == 0 : n % d.stride == 0) {
        // recorded steps from base to n, less one, within the block of K
        int slot;
        if (narrow) {
            const unsigned st = (unsigned)d.stride;
            const unsigned before = base > 0 ? (unsigned)(base - 1) / st + 1u : 0u;
            slot = (int)(((unsigned)n / st - before) % (unsigned)d.K);
        } else {
            const long long cnt = recorded_upto(n, d.stride) - recorded_upto(base - 1, d.stride);
            slot = (int)((cnt - 1) % d.K);
        }
        const bool flush = slot == d.K - 1;
        // this step's phasors: for the later steps of the block, and (every
        // CTA for itself) for the flush
        if (lb == 0 || flush) {
            const double tE = (double)n * d.dt;
            const double tH = tE + 0.5 * d.dt;
            const double dtw = (double)d.stride * d.dt;
            for (int q = threadIdx.x; q < 2 * d.nf; q += blockDim.x) {
                const int f = q % d.nf;
                const double t = (q < d.nf) ? tE : tH;
                double sn, cs;
                sincos(d.omega[f] * t, &sn, &cs);
                const float2 w = make_float2((float)(cs * dtw), (float)(sn * dtw));
                const long long at = ((long long)slot * 2 + (q / d.nf)) * d.nf + f;
                if (flush)
                    sw[at] = w;
                else
                    d.wst[at] = w;
            }
        }
        if (flush) {
            for (int q = threadIdx.x; q < (d.K - 1) * 2 * d.nf; q += blockDim.x) sw[q] = d.wst[q];
            __syncthreads();
        }
        const int total = d.ncomp * (int)d.ncell;
        for (int t = lb * kThreads + threadIdx.x; t < total; t += d.sblk * kThreads) {
            const int ci = t / (int)d.ncell;
            const int cell = t - ci * (int)d.ncell;
            const int kk = cell % d.nk;
            const int r = cell / d.nk;
            const int jj = r % d.nj;
            const int ii = r / d.nj;
            const int c = d.comps[ci];
            for (int b = 0; b < B; ++b) {
                const float v = (float)interp_sample<T>(e + (long long)b * e_block, h + (long long)b * h_block, g.vol,
                                                        g, d, c, d.i0 + ii, d.j0 + jj, d.k0 + kk);
                float* x = d.stage + ((long long)b * d.K * d.ncomp + ci) * d.ncell + cell;
                if (flush)
                    flush_cell(d, d.K, c < 3 ? 0 : 1, x, (long long)total, d.K - 1, v,
                               ((long long)(b * d.ncomp + ci) * d.nf) * d.ncell + cell, sw);
                else
                    x[(long long)slot * total] = v;
            }
        }
    }
    if (done) return;
    // The last CTA to finish advances the step counter: every CTA has read
    // it above, and the next launch in the stream starts after this one.
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd(ticket, 1u) == gridDim.x - 1) {
            *ticket = 0u;
            step[0] = n + 1;
            __threadfence();
        }
    }
}

// The first kc slots of one monitor, on request.
__global__ void __launch_bounds__(kThreads) k_dft_flush_forced(int B, DftDev d, int kc) {
    extern __shared__ float2 sw[];
    for (int q = threadIdx.x; q < kc * 2 * d.nf; q += blockDim.x) sw[q] = d.wst[q];
    __syncthreads();
    const long long per_b = (long long)d.ncomp * d.ncell;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < B * per_b;
         t += (long long)gridDim.x * blockDim.x) {
        const int b = (int)(t / per_b);
        const long long r = t % per_b;
        const int ci = (int)(r / d.ncell);
        const long long cell = r % d.ncell;
        flush_cell(d, kc, d.comps[ci] < 3 ? 0 : 1, d.stage + ((long long)b * d.K * d.ncomp + ci) * d.ncell + cell,
                   per_b, kc, 0.0f, ((long long)(b * d.ncomp + ci) * d.nf) * d.ncell + cell, sw);
    }
}

}  // namespace

int dft_blocks(long long work) {
    long long b = (work + kThreads - 1) / kThreads;
    if (b > 148 * 4) b = 148 * 4;
    return (int)(b < 1 ? 1 : b);
}

template <typename T>
void launch_dft_step(const T* e, const T* h, long long e_block, long long h_block, const Geom& g, int B,
                     const DftPack& pack, const DftDev* devs, int nmon, int nblocks, size_t smem, long long* step,
                     int done, unsigned* ticket, cudaStream_t s) {
    if (nmon <= kDftPack)
        k_dft_step<T, true>
            <<<nblocks, kThreads, smem, s>>>(e, h, e_block, h_block, g, B, pack, devs, nmon, step, done, ticket);
    else
        k_dft_step<T, false>
            <<<nblocks, kThreads, smem, s>>>(e, h, e_block, h_block, g, B, pack, devs, nmon, step, done, ticket);
}

void launch_dft_flush_forced(int B, const DftDev& d, int kc, cudaStream_t s) {
    const size_t smem = (size_t)kc * 2 * d.nf * sizeof(float2);
    k_dft_flush_forced<<<dft_blocks((long long)B * d.ncomp * d.ncell), kThreads, smem, s>>>(B, d, kc);
}

template void launch_dft_step<float>(const float*, const float*, long long, long long, const Geom&, int,
                                     const DftPack&, const DftDev*, int, int, size_t, long long*, int, unsigned*,
                                     cudaStream_t);
template void launch_dft_step<double>(const double*, const double*, long long, long long, const Geom&, int,
                                      const DftPack&, const DftDev*, int, int, size_t, long long*, int, unsigned*,
                                      cudaStream_t);

}  // namespace fitb
