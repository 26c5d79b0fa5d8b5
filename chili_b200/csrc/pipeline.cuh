// pipeline.cuh -- the phased form of the all-channel weight pass.
//
// Integrand::GenerateWeight (include/Channel/Integrand.hh:112-123) evaluated
// for a list of points in four kernels with small per-thread state, instead of
// one thread running every channel's inverse mapping from start to end:
//   k_pp_nodes     gathers the point's external momenta and sums the compound
//                  currents (one thread per point)
//   k_pp_items     every t-channel entry, decay propagator weight and
//                  two-body decay weight (one thread per point and item)
//   k_pp_chains    every t-channel chain's weight and last uniform (one thread
//                  per point and chain)
//   k_pp_channel   every channel's density and VEGAS weight (one thread per
//                  point and channel; the channel's uniforms come from the
//                  memo slots through its position map and stay in registers:
//                  DIMS is a compile-time constant)
//   k_pp_combine   per point, the combined weight in channel order, the
//                  integrand and the records of k_mc_weight.
// Intermediate values live in SoA buffers [slot][point] of one tile of points
// (stride m), so every access of a warp is coalesced and a tile's buffers
// stay in L2.
#pragma once

#include "phase_dev.cuh"

namespace chili_dev {



__global__ void __launch_bounds__(256) k_pp_nodes(const PointProgram *__restrict__ pp, const double *__restrict__ mom_soa,
                                                  long long mc, const int32_t *__restrict__ list,
                                                  const int32_t *__restrict__ ich_arr,
                                                  const long long *__restrict__ n_list, long long base,
                                                  double *__restrict__ node_soa, int32_t *__restrict__ ich_tile,
                                                  long long m) {
    pp_nodes_block(pp, mom_soa, mc, list, ich_arr, n_list, base, node_soa, ich_tile, m, blockIdx.x);
}


template <int KIND>
__global__ void __launch_bounds__(256, KIND == 2 ? 4 : 1) k_pp_items(const PointProgram *__restrict__ pp,
                                                  const double *__restrict__ node_soa,
                                                  const long long *__restrict__ n_list, long long base, long long m,
                                                  double *__restrict__ memo) {
    pp_items_block<KIND>(pp, node_soa, n_list, base, m, memo, blockIdx.x, blockIdx.y);
}

// Fills the (smin, smax)-only propagator terms of the point program with the
// device's own pow/atan, so that the shortcut in k_pp_items reproduces the
// full evaluation bit for bit.
__global__ void k_pp_prepare(PointProgram *__restrict__ pp) {
    const int k = threadIdx.x + blockIdx.x * blockDim.x;
    if (k < pp->n_dws) pp_prepare_entry(pp, k);
}


__global__ void __launch_bounds__(256) k_pp_chains(const PointProgram *__restrict__ pp,
                                                   const double *__restrict__ node_soa,
                                                   const long long *__restrict__ n_list, long long base, long long m,
                                                   double *__restrict__ memo, uint8_t *__restrict__ cfail) {
    pp_chains_block(pp, node_soa, n_list, base, m, memo, cfail, blockIdx.x, blockIdx.y);
}


// One block per (channel = blockIdx.x, range of `points` points =
// blockIdx.y): pp_channel_block.  The channels of a point range are
// consecutive blocks, so that the range's memo rows stay in L2 between them.
// A block holds one channel's tables in shared memory (TAB) while it works
// through its points; launch_channel picks the block and range sizes.  Bound
// by the latency of the memo loads (32 warps per SM at 64 registers) and by
// shared-memory bank conflicts.  Per iteration of 1e6 points: 2->4, 15 x 10
// searches per point, 0.43 ms; 2->6, 45 x 16 searches, 1.57 ms (the hinted
// binary searches this replaces: 0.58 and 4.89 ms).
template <int DIMS, bool TAB, int F, bool REC>
__global__ void __launch_bounds__(channel_max_threads(DIMS), DIMS > 16 ? 1 : 1024 / channel_max_threads(DIMS)) k_pp_channel(
    const PointProgram *__restrict__ pp, GridTables T, int bins, const double *__restrict__ memo,
    const uint8_t *__restrict__ cfail, const int32_t *__restrict__ ich_tile, const long long *__restrict__ n_list,
    long long base, long long m, Densities dens, double *__restrict__ vwv, void *__restrict__ own_out, int points) {
    extern __shared__ __align__(16) char smem[];
    const long long i0 = blockIdx.y * static_cast<long long>(points);
    const long long left = *n_list - base, end = left < m ? left : m;
    if (i0 >= end) return;
    const long long i1 = i0 + points < end ? i0 + points : end;
    pp_channel_block<DIMS, TAB, F, REC>(pp, T, bins, memo, cfail, ich_tile, m, dens, vwv, own_out, base, i0, i1,
                                        blockIdx.x, smem);
}

// Per point: 1 / sum_c alpha_c / dens_c / vw_c in channel order
// (Integrand.hh:118-122), the integrand and the value records.
__global__ void __launch_bounds__(256) k_pp_combine(const PointProgram *__restrict__ pp,
                                                    const double *__restrict__ alpha,
                                                    Densities dens, const double *__restrict__ vwv,
                                                    const double *__restrict__ node_soa,
                                                    const long long *__restrict__ n_list, long long base, long long m,
                                                    const IntegrandDesc *__restrict__ f, double *__restrict__ rec_val,
                                                    double *__restrict__ rec_wgt, uint8_t *__restrict__ rec_ok) {
    const long long i = blockIdx.x * 256ll + threadIdx.x;
    const long long r = base + i;
    if (i >= m || r >= *n_list) return;
    pp_combine_point(pp, alpha, dens, vwv, node_soa, m, i, r, f, rec_val, rec_wgt, rec_ok);
}

// ---------------------------------------- given or drawn points, every one
// Entry points that weight every point (chili_gpu_multichannel_weight,
// chili_gpu_generate) fill a tile's nodes themselves; the tile then takes the
// steps above.  One thread per point ran every channel from start to end
// before (4.6 and 5.7 ms per 1e6 points of 15 channels: ~50k instructions and
// an 8 KB local-memory frame per thread).
__device__ __forceinline__ bool aligned16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

// Tile of given momenta mom [point][leg][E, px, py, pz] from point `base` on:
// nodes, channels, the tile's point count, and zero uniforms for a point
// whose channel is none of the set's (x_own rows, where asked for).
__global__ void __launch_bounds__(256) k_pp_given(const PointProgram *__restrict__ pp, const double *__restrict__ mom,
                                                  const int32_t *__restrict__ ich, long long base, long long n,
                                                  long long m, double *__restrict__ node_soa,
                                                  int32_t *__restrict__ ich_tile, double *__restrict__ x_own,
                                                  long long *__restrict__ count) {
    const long long i = blockIdx.x * 256ll + threadIdx.x;
    if (i == 0) *count = n;
    if (i >= m || base + i >= n) return;
    const int ne = pp->n_ext, c = ich[base + i];
    const double *q = mom + (base + i) * ne * 4;
    if (aligned16(mom)) {
        for (int s = 0; s < ne; ++s) {
            const double2 a = reinterpret_cast<const double2 *>(q)[2 * s], b = reinterpret_cast<const double2 *>(q)[2 * s + 1];
            store_v4(node_soa, s, m, i, V4{a.x, a.y, b.x, b.y});
        }
    } else {
        for (int s = 0; s < ne; ++s) store_v4(node_soa, s, m, i, V4{q[4 * s], q[4 * s + 1], q[4 * s + 2], q[4 * s + 3]});
    }
    pp_compounds(pp, node_soa, m, i);
    ich_tile[i] = c;
    if (x_own && (c < 0 || c >= pp->nch))
        for (int d = 0; d < pp->ndims; ++d) x_own[(base + i) * pp->ndims + d] = 0.0;
}

// Tile of drawn points (counters ctr0 + base + i): channel, VEGAS map,
// FSMapper; nodes, the tile's channels and count (node_soa null: none of
// them), and the points' momenta and channels where asked for.  No PreProcess.
__global__ void __launch_bounds__(kFwdBlock, 3) k_pp_drawn(
    const PointProgram *__restrict__ pp, const ChannelProgram *__restrict__ progs, const double *__restrict__ grids,
    const double *__restrict__ cp, int dims, int bins, uint64_t seed, uint64_t ctr0, long long base, long long n,
    long long m, double *__restrict__ node_soa, int32_t *__restrict__ ich_tile, double *__restrict__ mom_out,
    int32_t *__restrict__ ch_out, long long *__restrict__ count) {
    const long long i = blockIdx.x * static_cast<long long>(kFwdBlock) + threadIdx.x;
    if (i == 0 && node_soa) *count = n;
    if (i >= m || base + i >= n) return;
    const int ne = pp->n_ext;
    V4 mom[CHILI_MAX_SLOTS];
    const int c = draw_point(progs, grids, cp, pp->nch, dims, bins, seed, ctr0 + base + i, nullptr, ne, mom);
    if (mom_out) {
        double *o = mom_out + (base + i) * ne * 4;
        if (aligned16(mom_out)) {
            for (int s = 0; s < ne; ++s) {
                reinterpret_cast<double2 *>(o)[2 * s] = make_double2(mom[s].e, mom[s].x);
                reinterpret_cast<double2 *>(o)[2 * s + 1] = make_double2(mom[s].y, mom[s].z);
            }
        } else {
            for (int s = 0; s < ne; ++s) {
                o[4 * s] = mom[s].e; o[4 * s + 1] = mom[s].x; o[4 * s + 2] = mom[s].y; o[4 * s + 3] = mom[s].z;
            }
        }
    }
    if (ch_out) ch_out[base + i] = c;
    if (!node_soa) return;  // no weights asked for
    ich_tile[i] = c;
    for (int s = 0; s < ne; ++s) store_v4(node_soa, s, m, i, mom[s]);
    pp_compounds(pp, node_soa, m, i);
}

// The combined weight of every tile point (f null; dens_out: the densities
// too, [point][channel]), or its value f w with non-finite values as 0 (event
// generation).
__global__ void __launch_bounds__(256) k_pp_weights(const PointProgram *__restrict__ pp,
                                                    const double *__restrict__ alpha, Densities dens,
                                                    const double *__restrict__ vwv,
                                                    const double *__restrict__ node_soa, long long base, long long n,
                                                    long long m, const IntegrandDesc *__restrict__ f,
                                                    double *__restrict__ dens_out, double *__restrict__ out) {
    const long long i = blockIdx.x * 256ll + threadIdx.x;
    if (i >= m || base + i >= n) return;
    const int nch = pp->nch;
    double w = pp_weight_sum(nch, alpha, dens, vwv, m, i, dens_out ? dens_out + (base + i) * nch : nullptr);
    if (f) {
        w = w == 0 ? 0 : eval_momenta_soa(f, node_soa, m, i, pp->n_ext) * w;
        if (!isfinite(w)) w = 0;
    }
    out[base + i] = w;
}

}  // namespace chili_dev
