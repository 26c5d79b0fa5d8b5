// mc_device.cuh -- types and device helpers shared by the kernels of
// libchili_b200 (kernels.cuh, pipeline.cuh, flow_phys.cuh): iteration
// accumulator and round records, the channel-selection rule, the checked
// grid map, the counter-based uniforms, the combined channel weight, the
// channel-weight update and the grid adaptation of one dimension.
#pragma once

#include <math_constants.h>

#include "channel_program.h"
#include "common.cuh"
#include "fsmapper.cuh"
#include "grid.cuh"
#include "integrands.cuh"

namespace chili_dev {

constexpr int kFwdBlock = 256;
constexpr int kWgtBlock = 128;
constexpr int kVegasBlock = 256;

// Iteration accumulator of a multichannel iteration (device resident).
struct IterAcc {
    double st[6];      // n, min, max, sum, sum2, n_finite
    double nan_count;  // NaN-value retries
    double nonfinite;  // dropped alpha-training terms (guard mode)
    double wmax;       // max value
    double dropped;    // histogram adds before the histogram (dim 0, FindBin SIZE_MAX)
    double rejected_pre;
    double pad;
    double atrain[CHILI_MAX_CHANNELS];
};

// Round control written by k_mc_scan / k_mc_finalize, read by the host.
struct RoundCtl {
    long long cut;        // counters consumed by this round
    long long n_acc;      // PreProcess-accepted points before the cut
    long long nan_round;  // of those, NaN retries
    long long pad;
};

constexpr int kPartFixed = 10;  // n, min, max, sum, sum2, nfin, nan, nonfin, wmax, dropped

// A record's histogram bins: dims halfwords 8 (FindBin + 1) in the record's
// channel (the byte offsets the channel step reads its widths at), then the
// channel, in bin_rec_vecs(dims) 16-byte words (one row per
// record, so that the channel step writes a point's bins in two or three
// stores and the accumulation reads them in as many).
__host__ __device__ inline int bin_rec_vecs(int dims) { return (dims + 8) / 8; }

// fn(s) for every dimension of record r: the flat histogram slot s of the
// record's channel the way Integrand::AddTrainData indexes it
// (Integrand.hh:91-95; a FindBin of SIZE_MAX wraps to the previous
// dimension's last bin), -1 where it lies before the histogram.
template <class Fn>
__device__ __forceinline__ void for_each_train_slot(const uint4 *__restrict__ rec_bins, long long r, int dims, int bins,
                                                    Fn fn) {
    const int nv = bin_rec_vecs(dims);
    const uint4 *p = rec_bins + r * nv;
    const int base = static_cast<int>(reinterpret_cast<const uint16_t *>(p)[dims]) * dims * bins;
    for (int j = 0; j < nv; ++j) {
        const uint4 v = p[j];
        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int h = 0; h < 8; ++h) {
            const int d = 8 * j + h;
            if (d < dims) {
                const int s = d * bins + static_cast<int>(((w[h >> 1] >> (16 * (h & 1))) & 0xffffu) >> 3) - 1;
                fn(s >= 0 ? base + s : -1);
            }
        }
    }
}

// libstdc++ lower_bound over cp[0..n) (probe order of bits/stl_algobase.h).
__device__ __forceinline__ int lower_bound_d(const double *__restrict__ a, int n, double v) {
    int first = 0, len = n;
    while (len > 0) {
        const int half = len >> 1;
        const int mid = first + half;
        if (__ldg(a + mid) < v) {
            first = mid + 1;
            len = len - half - 1;
        } else {
            len = half;
        }
    }
    return first;
}

// Random::SelectIndex == std::discrete_distribution (Random.hh:43-45): the
// index of the first cumulative probability not below v.
__device__ __forceinline__ int select_channel(const double *__restrict__ cp, int nch, double v) {
    if (nch < 2) return 0;
    const int i = lower_bound_d(cp, nch, v);
    return i < nch ? i : nch - 1;
}

// Forward grid map with the bin index checked: returns false (x untouched
// beyond the failing dimension) when a uniform is outside [0, 1).
__device__ __forceinline__ bool grid_map_checked(const double *__restrict__ g, int dims, int bins, double *x,
                                                 double &jac) {
    jac = 1.0;
    const double fb = static_cast<double>(bins);
    for (int d = 0; d < dims; ++d) {
        const double pos = __dmul_rn(x[d], fb);
        if (!(pos >= 0.0 && pos < fb)) return false;
        double whole;
        const int idx = floor_index(pos, whole);
        const double loc = __dsub_rn(pos, whole);
        const double *e = g + d * (bins + 1);
        const double left = __ldg(e + idx);
        const double size = __dsub_rn(__ldg(e + idx + 1), left);
        x[d] = __dadd_rn(left, __dmul_rn(loc, size));
        jac = __dmul_rn(jac, __dmul_rn(size, fb));
    }
    return true;
}

__device__ __forceinline__ void load_uniforms(uint64_t seed, uint64_t k, const double *__restrict__ u_in,
                                              int n, double *out) {
    if (u_in) {
        for (int j = 0; j < n; ++j) out[j] = __ldg(u_in + k * n + j);
    } else {
        for (int q = 0; 2 * q < n; ++q) {
            double a, b;
            uniform_pair(seed, k, kStreamPoints, static_cast<uint32_t>(q), a, b);
            out[2 * q] = a;
            if (2 * q + 1 < n) out[2 * q + 1] = b;
        }
    }
}

// One drawn point: its channel's FSMapper momenta (slots mom) from the
// uniforms of counter k (or row k of u_in), through the channel's VEGAS grid;
// all NaN when a uniform lies outside [0, 1).  Returns the channel.
// (The uniforms are made before the FSMapper: made where it consumes them,
// lanes of different channels made them at different times, 1.16x slower.)
__device__ __forceinline__ int draw_point(const ChannelProgram *__restrict__ progs, const double *__restrict__ grids,
                                          const double *__restrict__ cp, int nch, int dims, int bins, uint64_t seed,
                                          uint64_t k, const double *__restrict__ u_in, int n_ext, V4 *mom) {
    double r[CHILI_MAX_DIMS + 1], jac;
    load_uniforms(seed, k, u_in, dims + 1, r);
    const int c = select_channel(cp, nch, r[dims]);
    if (grid_map_checked(grids + static_cast<size_t>(c) * dims * (bins + 1), dims, bins, r, jac)) {
        double m2[CHILI_MAX_SLOTS];
        fs_generate(progs + c, r, mom, m2);
    } else {
        for (int s = 0; s < n_ext; ++s) mom[s] = V4{CUDART_NAN, CUDART_NAN, CUDART_NAN, CUDART_NAN};
    }
    return c;
}

// ------------------------------------------------- shared by several kernels
// Integrand::GenerateWeight (Integrand.hh:112-123) for one point.  The
// uniform buffer x is shared by all channels and not cleared between them,
// as the reference's _rans; the chosen channel's copy lands in xs.
__device__ __forceinline__ double combined_weight(const ChannelProgram *__restrict__ progs,
                                                  const double *__restrict__ grids, const double *__restrict__ alpha,
                                                  int nch, int dims, int bins, int ich, V4 *mom, double *x,
                                                  double *xs, double *dens, int dens_stride) {
    for (int d = 0; d < dims; ++d) x[d] = 0.0;
    double acc = 0;
    const size_t gsz = static_cast<size_t>(dims) * (bins + 1);
    const double before = edge_before_table(dims, bins);
    for (int c = 0; c < nch; ++c) {
        const double dc = fs_weight(progs + c, mom, x);
        if (c == ich)
            for (int d = 0; d < dims; ++d) xs[d] = x[d];
        const double vw = grid_weight(grids + c * gsz, dims, bins, x, before);
        acc += __ldg(alpha + c) / dc / vw;
        if (dens) dens[static_cast<size_t>(c) * dens_stride] = dc;
    }
    return 1.0 / acc;
}


// MultiChannel::Adapt and MaxDifference (MultiChannel.cc:109-154; mode 1),
// then the cumulative table of std::discrete_distribution, by one block.  The
// order-dependent sums run in thread 0 over shared memory; the powers, the
// quotients and the largest difference (a maximum, independent of order) in
// parallel: one thread for all of it took 17 us at 15 channels.
__device__ __forceinline__ void alpha_update(double *__restrict__ alpha, double *__restrict__ best,
                                             double *__restrict__ min_diff, double *__restrict__ cp,
                                             const double *__restrict__ train, int nch, double beta, double min_alpha,
                                             int mode) {
    __shared__ double v_s[CHILI_MAX_CHANNELS], red_s[32], sum_s;
    const int t = threadIdx.x, nt = blockDim.x;
    __syncthreads();
    if (mode == 1) {
        for (int i = t; i < nch; i += nt) v_s[i] = alpha[i] * pow(train[i], beta);
        double mx = 0;  // a NaN difference never compares larger
        for (int q = t; q < nch * nch; q += nt) {
            const int i = q / nch, j = q - i * nch;
            if (j > i) mx = std_max(mx, fabs(train[i] - train[j]));
        }
        mx = warp_max(mx);
        if ((t & 31) == 0) red_s[t >> 5] = mx;
        __syncthreads();
        if (t == 0) {
            double s = 0;
            for (int i = 0; i < nch; ++i) s += v_s[i];
            sum_s = s;
        }
        __syncthreads();
        for (int i = t; i < nch; i += nt)
            if (v_s[i] != 0) v_s[i] = std_max(v_s[i] / sum_s, min_alpha);
        __syncthreads();
        if (t == 0) {
            double s = 0;
            for (int i = 0; i < nch; ++i)
                if (v_s[i] != 0) s += v_s[i];
            sum_s = s;
        }
        __syncthreads();
        for (int w = 0; w < (nt + 31) / 32; ++w) mx = std_max(mx, red_s[w]);
        const bool better = mx < *min_diff;
        for (int i = t; i < nch; i += nt) {
            const double a = v_s[i] / sum_s;
            alpha[i] = a;
            v_s[i] = a;
            if (better) best[i] = a;
        }
        __syncthreads();  // every thread has read min_diff
        if (t == 0 && better) *min_diff = mx;
    } else {
        for (int i = t; i < nch; i += nt) v_s[i] = alpha[i];
        __syncthreads();
    }
    if (nch >= 2) {
        if (t == 0) {
            double s = 0;
            for (int i = 0; i < nch; ++i) s += v_s[i];
            sum_s = s;
        }
        __syncthreads();
        for (int i = t; i < nch; i += nt) v_s[i] = v_s[i] / sum_s;
        __syncthreads();
        if (t == 0) {
            double c = 0;
            for (int i = 0; i < nch; ++i) {
                c = (i == 0) ? v_s[i] : c + v_s[i];
                cp[i] = c;
            }
            cp[nch - 1] = 1.0;
        }
    }
}

// Shared-memory bytes of the adaptation of one row: the factors (doubles)
// and the bins that the edges fall in (halfwords).
__host__ __device__ constexpr size_t adapt_scratch_bytes(int bins) {
    return sizeof(double) * (static_cast<size_t>(bins) + (bins + 3) / 4);
}

// AdaptiveMap::Adapt (AdaptiveMap.cc:67-125) of dimension d of grid c by one
// block (WARP false) or by one warp (WARP true: the lanes of the calling
// warp); tmp: adapt_scratch_bytes(bins) of shared memory of its own.  The
// order-dependent sums and the walk over the factors run serially in thread
// (lane) 0 in the reference's order; smoothing, importance factors and the
// new edges in parallel.  Computing the edges inside the walk made every one
// of its steps wait for two edge loads and a division: 41 us for the 150 rows
// of 100 bins of the 2->4 set.
template <bool WARP>
__device__ __forceinline__ void grid_adapt_impl(const double *__restrict__ g_old, double *__restrict__ g_new, int dims,
                                                int bins, double alpha, const double *__restrict__ train,
                                                int skip_zero, int *__restrict__ status, int d, int c, double *tmp) {
    const int tid = WARP ? static_cast<int>(threadIdx.x & 31) : static_cast<int>(threadIdx.x);
    const int nthr = WARP ? 32 : static_cast<int>(blockDim.x);
    auto sync = [] {
        if (WARP) __syncwarp();
        else __syncthreads();
    };
    uint16_t *at = reinterpret_cast<uint16_t *>(tmp + bins);  // factors used up to each new edge
    const double *T = train + static_cast<size_t>(c) * dims * bins;
    const double *E = g_old + static_cast<size_t>(c) * dims * (bins + 1);
    double *EN = g_new + static_cast<size_t>(c) * dims * (bins + 1);
    const double *Ed = E + d * (bins + 1);
    double *ENd = EN + d * (bins + 1);
    if (skip_zero) {
        int nz = 0;
        for (int k = tid; k < dims * bins; k += nthr) nz |= (T[k] != 0);
        nz = WARP ? __any_sync(0xffffffffu, nz) : __syncthreads_or(nz);
        if (!nz) {
            for (int k = tid; k <= bins; k += nthr) ENd[k] = Ed[k];
            return;
        }
    }
    const double *o = T + d * bins;
    for (int b = tid; b < bins; b += nthr) {
        double s;
        if (b == 0) s = (o[0] + o[1]) / 2;
        else if (b == bins - 1) s = (o[bins - 2] + o[bins - 1]) / 2;
        else s = ((o[b - 1] + o[b]) + o[b + 1]) / 3;
        tmp[b] = s;
    }
    sync();
    double norm = 0;
    if (WARP) {
        if (tid == 0)
            for (int b = 0; b < bins; ++b) norm = (b == 0) ? tmp[0] : norm + tmp[b];
        norm = __shfl_sync(0xffffffffu, norm, 0);
    } else {
        __shared__ double norm_s;
        if (tid == 0) {
            double nm = 0;
            for (int b = 0; b < bins; ++b) nm = (b == 0) ? tmp[0] : nm + tmp[b];
            norm_s = nm;
        }
        __syncthreads();
        norm = norm_s;
    }
    if (norm == 0) {  // the reference leaves this dimension of new_hist at zero
        for (int k = tid; k <= bins; k += nthr) ENd[k] = 0.0;
        return;
    }
    for (int b = tid; b < bins; b += nthr) {
        if (tmp[b] != 0) {
            const double r = tmp[b] / norm;
            tmp[b] = pow((r - 1.0) / log(r), alpha);
        }
    }
    sync();
    if (tid == 0) {
        double avg = 0;
        for (int b = 0; b < bins; ++b) avg += tmp[b];
        avg /= static_cast<double>(bins);
        double cbin = 0, next = tmp[0];
        int ibin = 0;
        int bad = 0;
        ENd[0] = 0.0;
        for (int nb = 1; nb < bins; ++nb) {
            while (cbin < avg && ibin < bins) {
                cbin += next;
                ++ibin;
                next = tmp[ibin < bins ? ibin : bins - 1];
            }
            if (cbin < avg || ibin == 0) bad = 1;  // the reference would read outside the histogram
            cbin -= avg;
            ENd[nb] = cbin;  // what of the last factor lies beyond the edge, until the edges are computed
            at[nb] = static_cast<uint16_t>(ibin);
        }
        ENd[bins] = 1.0;
        if (bad) atomicOr(status, 1);
    }
    sync();
    for (int nb = 1 + tid; nb < bins; nb += nthr) {
        const int ibin = at[nb];
        const int flat_prev = d * (bins + 1) + ibin - 1;
        const double prev = flat_prev >= 0 ? E[flat_prev] : CUDART_NAN;
        const double curr = Ed[ibin];
        const double delta = (curr - prev) * ENd[nb];
        const double t = ibin > 0 ? tmp[ibin - 1] : CUDART_NAN;
        ENd[nb] = curr - delta / t;
    }
    sync();
}

__device__ __forceinline__ void grid_adapt_block(const double *__restrict__ g_old, double *__restrict__ g_new, int dims,
                                                 int bins, double alpha, const double *__restrict__ train, int skip_zero,
                                                 int *__restrict__ status, int d, int c, double *tmp) {
    grid_adapt_impl<false>(g_old, g_new, dims, bins, alpha, train, skip_zero, status, d, c, tmp);
}

}  // namespace chili_dev
