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
// All monitors share one launch per step (k_dft_step), or, where one of them
// has many samples, a launch that stages and one that flushes.
#include "fitb_common.cuh"

#include <algorithm>
#include <type_traits>

namespace fitb {

namespace {

constexpr int kMaxK = 32;
constexpr int kThreads = 256;
constexpr int kResident = 148 * 4;  // CTAs of 64 registers a thread that the chip holds

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
// the bins of one cell-component: bins bi + f * ncell, phasors sw.  FULL: a
// block of kMaxK samples (up to 96 frequencies), whose sums need no comparison
// per sample and frequency (six components of 0.9 M cells, 64 frequencies: 159
// us per step against 254 with them).
template <bool FULL>
__device__ __forceinline__ void flush_cell(const DftDev& d, int kc, int tsel, const float* x, long long xs, int n_st,
                                           float last, long long bi, const float2* sw) {
    float v[kMaxK];
#pragma unroll
    for (int s = 0; s < kMaxK; ++s) v[s] = s < n_st ? x[s * xs] : (s == kc - 1 ? last : 0.0f);
    sw += tsel * d.nf;
    for (int f = 0; f < d.nf; ++f, bi += d.ncell, ++sw) {
        float2 acc = d.bins[bi], cm;
        if (d.kahan) cm = d.cmp[bi];
        float re = 0.0f, im = 0.0f;
#pragma unroll
        for (int s = 0; s < kMaxK; ++s) {
            if (FULL || s < kc) {
                const float2 w = sw[s * 2 * d.nf];
                re = fmaf(w.x, v[s], re);
                im = fmaf(w.y, v[s], im);
            }
        }
        if (d.kahan) {
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

// One step of every monitor: PARTS = both, or the staging and the flush as
// launches of their own.  The step counter is *step - done: done = 1 when an
// earlier kernel of the step has advanced it; otherwise the last CTA to finish
// (of the flush) does, through `ticket`.
// Both in one launch saves the flush's, which is empty on K - 1 of K steps, and
// gives a thread one sample of one field set: on a 97 x 104 x 89 mesh with
// three planes of 16 frequencies 4.9 us per step against 8.4 in two launches;
// eight sets of a 64 x 56 plane with 64 frequencies 7.1 us against 16.7 (and 44
// where a thread walked its cell's sets).  From about 0.6 M samples on, two
// launches of loops that hold 64 registers each: the staging of a cell's sets
// shares its indexing, and no CTA is too short for its descriptor's latency
// (three components of 0.9 M cells, eight frequencies: 39 us with one field set
// and 105 with four; as one launch 48 and 186).
// The launch is short, so its chain counts: up to kDftPack descriptors travel
// as kernel arguments (else a block's first loads are a descriptor from HBM or
// L2, one after the other per monitor), and the slot arithmetic is 32-bit
// while the step count is.
constexpr int kStage = 1, kFlush = 2;
template <typename T, int PARTS, bool PACK>
__global__ void __launch_bounds__(kThreads, 4)
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
        // this step's phasors: for the flush to come, and, where it is in this
        // launch, every CTA for itself
        constexpr bool kBoth = PARTS == (kStage | kFlush);
        const bool own = kBoth && flush;
        if ((PARTS & kStage) && (lb == 0 || own)) {
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
                if (own)
                    sw[at] = w;
                else
                    d.wst[at] = w;
            }
        }
        if ((PARTS & kFlush) && flush) {
            for (int q = threadIdx.x; q < (kBoth ? d.K - 1 : d.K) * 2 * d.nf; q += blockDim.x) sw[q] = d.wst[q];
            __syncthreads();
        }
        const int per_set = d.ncomp * (int)d.ncell;
        const int t0 = lb * kThreads + threadIdx.x;
        const auto sample = [&](int b, int r) {  // component and cell r of field set b
            const int ci = r / (int)d.ncell;
            const int cell = r - ci * (int)d.ncell;
            const int kk = cell % d.nk;
            const int rr = cell / d.nk;
            const int jj = rr % d.nj;
            const int ii = rr / d.nj;
            return (float)interp_sample<T>(e + (long long)b * e_block, h + (long long)b * h_block, g.vol, g, d,
                                           d.comps[ci], d.i0 + ii, d.j0 + jj, d.k0 + kk);
        };
        const auto add = [&](int b, int r, int n_st, float last) {
            const int ci = r / (int)d.ncell;
            const auto go = [&](auto full) {
                flush_cell<decltype(full)::value>(
                    d, d.K, d.comps[ci] < 3 ? 0 : 1, d.stage + (long long)b * d.K * per_set + r, per_set, n_st, last,
                    (long long)(b * d.ncomp + ci) * d.nf * d.ncell + (r - ci * (int)d.ncell), sw);
            };
            if (d.K == kMaxK)
                go(std::true_type());
            else
                go(std::false_type());
        };
        if constexpr (kBoth) {
            if (t0 < B * per_set) {
                const int b = t0 / per_set, r = t0 - b * per_set;
                const float v = sample(b, r);
                if (flush)
                    add(b, r, d.K - 1, v);
                else
                    d.stage[((long long)b * d.K + slot) * per_set + r] = v;
            }
        } else if constexpr (PARTS == kStage) {
            for (int r = t0; r < per_set; r += d.sblk * kThreads)
                for (int b = 0; b < B; ++b) d.stage[((long long)b * d.K + slot) * per_set + r] = sample(b, r);
        } else if (flush) {
            for (int t = t0; t < B * per_set; t += d.sblk * kThreads) {
                const int b = t / per_set;
                add(b, t - b * per_set, d.K, 0.0f);
            }
        }
    }
    if (PARTS == kStage) return;
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
        flush_cell<false>(d, kc, d.comps[ci] < 3 ? 0 : 1, d.stage + ((long long)b * d.K * d.ncomp + ci) * d.ncell + cell,
                   per_b, kc, 0.0f, ((long long)(b * d.ncomp + ci) * d.nf) * d.ncell + cell, sw);
    }
}

}  // namespace

bool dft_one_launch(const DftDev& d, int B) {
    return (long long)B * d.ncomp * d.ncell <= 4LL * kResident * kThreads;
}

int dft_blocks(long long work, bool one_launch) {
    const long long n = (work + kThreads - 1) / kThreads;
    return (int)std::max(1LL, one_launch ? n : std::min<long long>(n, kResident));
}

template <typename T>
int launch_dft_step(const T* e, const T* h, long long e_block, long long h_block, const Geom& g, int B,
                    const DftPack& pack, const DftDev* devs, int nmon, int nblocks, size_t smem, bool one_launch,
                    long long* step, int done, unsigned* ticket, cudaStream_t s) {
    const auto go = [&](auto k, size_t sm) {
        k<<<nblocks, kThreads, sm, s>>>(e, h, e_block, h_block, g, B, pack, devs, nmon, step, done, ticket);
    };
    const bool packed = nmon <= kDftPack;
    if (one_launch) {
        packed ? go(k_dft_step<T, kStage | kFlush, true>, smem) : go(k_dft_step<T, kStage | kFlush, false>, smem);
        return 1;
    }
    packed ? go(k_dft_step<T, kStage, true>, 0) : go(k_dft_step<T, kStage, false>, 0);
    packed ? go(k_dft_step<T, kFlush, true>, smem) : go(k_dft_step<T, kFlush, false>, smem);
    return 2;
}

void launch_dft_flush_forced(int B, const DftDev& d, int kc, cudaStream_t s) {
    const size_t smem = (size_t)kc * 2 * d.nf * sizeof(float2);
    k_dft_flush_forced<<<dft_blocks((long long)B * d.ncomp * d.ncell, false), kThreads, smem, s>>>(B, d, kc);
}

#define FITB_INST(T)                                                                                                \
    template int launch_dft_step<T>(const T*, const T*, long long, long long, const Geom&, int, const DftPack&,      \
                                    const DftDev*, int, int, size_t, bool, long long*, int, unsigned*, cudaStream_t);
FITB_INST(float)
FITB_INST(double)
#undef FITB_INST

}  // namespace fitb
