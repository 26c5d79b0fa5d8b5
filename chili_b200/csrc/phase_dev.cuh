// phase_dev.cuh -- device functions of the phased weight pass and of the
// ordered compaction, with explicit block coordinates, shared by the
// kernels of one launch per step (pipeline.cuh, kernels.cuh) and by the
// grouped launches of the batched integrands (batch.cu), where one launch
// covers the pieces of many tasks.
#pragma once

#include <type_traits>

#include "channel_program.h"
#include "common.cuh"
#include "fsmapper.cuh"
#include "grid.cuh"
#include "integrands.cuh"
#include "mc_device.cuh"

namespace chili_dev {

// Rows of a tile's SoA buffers: element i of row r of stride m.  The row's
// offset is one 32 x 32 -> 64 bit multiply-add on the element's address (rows
// stay below 2^32 bytes: a tile or chunk has at most 2^24 points); with 64-bit
// strides the addresses took a tenth of the item kernels' instructions.
template <class T>
__device__ __forceinline__ T *soa_at(T *p, int r, long long m, long long i) {
    using Byte = std::conditional_t<std::is_const_v<T>, const char, char>;
    return reinterpret_cast<T *>(reinterpret_cast<Byte *>(p + i) +
                                 static_cast<unsigned long long>(static_cast<unsigned>(m) * 8u) *
                                     static_cast<unsigned>(r));
}
__device__ __forceinline__ V4 load_v4(const double *__restrict__ soa, int node, long long m, long long i) {
    const double *p = soa_at(soa, 4 * node, m, i);
    return V4{*p, *soa_at(p, 1, m, 0), *soa_at(p, 2, m, 0), *soa_at(p, 3, m, 0)};
}
__device__ __forceinline__ void store_v4(double *__restrict__ soa, int node, long long m, long long i, V4 v) {
    double *p = soa_at(soa, 4 * node, m, i);
    *p = v.e;
    *soa_at(p, 1, m, 0) = v.x;
    *soa_at(p, 2, m, 0) = v.y;
    *soa_at(p, 3, m, 0) = v.z;
}

// The compound nodes of tile point i, summed as the reference's tmp_mom, its
// external nodes being stored.
__device__ __forceinline__ void pp_compounds(const PointProgram *__restrict__ pp, double *__restrict__ node_soa,
                                             long long m, long long i) {
    const int ne = pp->n_ext, nn = pp->n_nodes;
    for (int s = ne; s < nn; ++s)
        store_v4(node_soa, s, m, i, load_v4(node_soa, pp->node_a[s], m, i) + load_v4(node_soa, pp->node_b[s], m, i));
}

// Nodes of point i = list[i]: externals copied from the chunk's momenta
// (mom_soa, stride mc), then the compounds.
__device__ __forceinline__ void pp_nodes_block(const PointProgram *__restrict__ pp, const double *__restrict__ mom_soa,
                                               long long mc, const int32_t *__restrict__ list,
                                               const int32_t *__restrict__ ich_arr,
                                               const long long *__restrict__ n_list, long long base,
                                               double *__restrict__ node_soa, int32_t *__restrict__ ich_tile,
                                               long long m, long long bx) {
    const long long i = bx * 256ll + threadIdx.x;  // tile-local point
    if (i >= m || base + i >= *n_list) return;
    const long long k = list[base + i];
    ich_tile[i] = ich_arr[k];
    for (int s = 0; s < pp->n_ext; ++s) store_v4(node_soa, s, m, i, load_v4(mom_soa, s, mc, k));
    pp_compounds(pp, node_soa, m, i);
}

// One thread per (point, item): items 0..n_tents-1 are t-channel entries
// (Channel.cc:160-186), then decay weights (Channel.cc:83-113), then two-body
// decays (Channel.cc:222-237).
// KIND selects the item type (0 t-entries, 1 decay weights, 2 two-body
// decays), so that each type gets its own register allocation; the two-body
// decays (80 registers unbounded) are held to 64 for four resident blocks
// per SM (2.3% faster items on the 2->4 workload than three).
// Block (bx = item of this kind, by = point block).  Bound by instruction
// issue (70-78% busy, FP64 pipe 44-57%): about 565, 500 and 880 instructions
// per item.  Quotients by constants of the set and by shared divisors are
// multiplications with a correction (div_by), the two-body decays leave out
// what the reference axis makes zero, roots that cannot matter are not taken:
// the results are those of the plain expressions, bit for bit.  Per 1e6
// points: 2->4 0.76 -> 0.61 ms, 2->6 1.79 -> 1.44 ms (three kernels).
template <int KIND>
__device__ __forceinline__ void pp_items_block(const PointProgram *__restrict__ pp,
                                               const double *__restrict__ node_soa,
                                               const long long *__restrict__ n_list, long long base, long long m,
                                               double *__restrict__ memo, int bx, long long by) {
    const long long i = by * 256ll + threadIdx.x;  // tile-local point
    if (i >= m || base + i >= *n_list) return;
    // consecutive blocks: items of the same points (L2 reuse)
    int item = bx + (KIND >= 1 ? pp->n_tents : 0) + (KIND >= 2 ? pp->n_dws : 0);
    const double sqrts = pp->sqrts, ptmax = pp->ptmax;
    if (KIND == 0 && item < pp->n_tents) {
        const int t = item;
        const double ptmin = pp->tent_ptmin[t];
        const V4 q = load_v4(node_soa, pp->tent_node[t], m, i);
        const double pt = sqrt(pt2(q));
        const double f2 = 2 * ptmin + pt;
        double *o = soa_at(memo, pp->memo_tent + 5 * t, m, i);
        *o = div_by(div_by(pt * ptmax * 0.5, ptmin, pp->tent_rptmin[t]), 2 * ptmin + ptmax, pp->tent_rsum[t]) * (f2 * f2);
        *soa_at(o, 2, m, 0) = pt * (ptmax + 2 * ptmin) / (ptmax * (pt + 2 * ptmin));
        double etamax = sqrts * 0.5 / pt;
        etamax = log(etamax + sqrt(etamax * etamax - 1));
        etamax = isnan(etamax) ? 99 : etamax;
        etamax = std_min(etamax, pp->tent_etacut[t]);
        *soa_at(o, 1, m, 0) = 2 * etamax * 2 * kPi;
        const double y = rapidity(q);
        if (pp->tent_y[t] >= 0) *soa_at(memo, pp->tent_y[t], m, i) = y;  // some chain's last node
        *soa_at(o, 3, m, 0) = (y / etamax + 1) * 0.5;
        *soa_at(o, 4, m, 0) = div_by(phi_0_2pi(q) * 0.5, kPi, kRcpPi);
        return;
    }
    item -= pp->n_tents;
    if (KIND == 1 && item < pp->n_dws) {
        const int k = item;
        const double ma = fabs(mass2(load_v4(node_soa, pp->dw_c1[k], m, i)));
        const double mb = fabs(mass2(load_v4(node_soa, pp->dw_c2[k], m, i)));
        const double s = mass2(load_v4(node_soa, pp->dw_node[k], m, i));
        double u, w, smin = pp->dw_smin_c[k];
        // (sqrt ma + sqrt mb)^2 <= 2 (ma + mb): below the cut without the roots
        if (!(2.0000001 * (ma + mb) < smin)) {
            const double r = sqrt(ma) + sqrt(mb);
            smin = std_max(std_max(r * r, pp->dw_smin2[k]), pp->dw_cut[k]);
        }
        if (smin == pp->dw_smin_c[k]) {  // the usual case: smin-only terms precomputed
            w = pp->dw_massless[k] ? massless_prop_weight_c(0.99, pp->dw_t1[k], pp->dw_t2[k], pp->dw_wce[k],
                                                            pp->dw_rspan[k], s, u)
                                   : massive_prop_weight_c(pp->dw_mass[k], pp->dw_width[k], pp->dw_t1[k],
                                                           pp->dw_t2[k], pp->dw_rspan[k], pp->dw_rmw[k], s, u);
        } else {
            w = pp->dw_massless[k] ? massless_prop_weight(0.99, smin, pp->dw_smax[k], s, u)
                                   : massive_prop_weight(pp->dw_mass[k], pp->dw_width[k], smin, pp->dw_smax[k], s, u);
        }
        double *o = soa_at(memo, pp->memo_dw + 2 * k, m, i);
        *o = w;
        *soa_at(o, 1, m, 0) = u;
        return;
    }
    item -= pp->n_dws;
    if (KIND == 2 && item < pp->n_sws) {
        const int k = item;
        double r1, r2;
        const double w = schannel_weight(load_v4(node_soa, pp->sw_a[k], m, i), load_v4(node_soa, pp->sw_b[k], m, i),
                                         r1, r2);
        double *o = soa_at(memo, pp->memo_sw + 3 * k, m, i);
        *o = w;
        *soa_at(o, 1, m, 0) = r1;
        *soa_at(o, 2, m, 0) = r2;
    }
}

// One thread per (point, chain): WgtTChan's weight and last uniform
// (Channel.cc:160-202), with the entries' factors and the last node's rapidity
// taken from the memo.  Issue-bound (81%, mostly logarithms and exponentials);
// per 1e6 points 2->4 0.29 -> 0.25 ms, 2->6 1.05 -> 0.94 ms with the shared
// rapidity, div_by and 32-bit row strides.
__device__ __forceinline__ void pp_chains_block(const PointProgram *__restrict__ pp,
                                                const double *__restrict__ node_soa,
                                                const long long *__restrict__ n_list, long long base, long long m,
                                                double *__restrict__ memo, uint8_t *__restrict__ cfail, int bx,
                                                long long by) {
    const long long i = by * 256ll + threadIdx.x;  // tile-local point
    if (i >= m || base + i >= *n_list) return;
    const int c = bx;  // consecutive blocks: chains of the same points
    const double sqrts = pp->sqrts;
    double wt = kTwoPi;
    V4 psum{0., 0., 0., 0.};
    const int len = pp->chain_len[c];
    for (int e = 0; e < len; ++e) {
        const int t = pp->chain_tent[c][e];
        const double *tm = soa_at(static_cast<const double *>(memo), pp->memo_tent + 5 * t, m, i);
        wt *= pp->inv16pi3;
        wt *= *tm;
        wt *= *soa_at(tm, 1, m, 0);
        psum = psum + load_v4(node_soa, pp->tent_node[t], m, i);
    }
    const V4 q = load_v4(node_soa, pp->chain_last[c], m, i);
    const double mjets2 = mass2(psum);
    const double yjets = rapidity(psum);
    const double ptj2 = pt2(psum);
    const double qt = sqrt(mass2(q) + ptj2);
    const double mt = sqrt(mjets2 + ptj2);
    // the last node's rapidity, where a t-channel entry has computed it
    const int ys = pp->chain_y[c];
    const double yv = ys >= 0 ? *soa_at(static_cast<const double *>(memo), ys, m, i) : rapidity(q);
    const double sq = sqrts / qt, ms = div_by(mt, sqrts, pp->rsqrts);
    const double ymin = -log(sq * (1 - ms * exp(-yjets)));
    const double ymax = log(sq * (1 - ms * exp(yjets)));
    const double dely = ymax - ymin;
    double *o = soa_at(memo, pp->memo_chain + 2 * c, m, i);
    const bool fail = isnan(ymax) || isnan(ymin);
    *o = fail ? 0 : wt * div_by(div_by(dely, sqrts, pp->rsqrts), sqrts, pp->rsqrts);
    *soa_at(o, 1, m, 0) = fail ? 0 : (yv - ymin) / dely;
    cfail[c * m + i] = fail;
}

// Pair Breit-Wigner / t-channel integrand reading the externals from the
// node buffer (same arithmetic as eval_momenta).
__device__ __forceinline__ double eval_momenta_soa(const IntegrandDesc *__restrict__ f,
                                                   const double *__restrict__ node_soa, long long m, long long i,
                                                   int n_ext) {
    if (f->kind != CHILI_FUNC_PROPAGATOR && f->kind != CHILI_FUNC_PROPAGATOR_TOP2) return 1.0;
    const bool top2 = f->kind == CHILI_FUNC_PROPAGATOR_TOP2;
    const double mm = f->p[0], g = f->p[1], mt = f->p[2];
    const double m2 = mm * mm, mw2 = mm * mm * g * g, mt2 = mt * mt;
    double sum = 0, big1 = 0, big2 = 0;
    for (int a = 2; a < n_ext; ++a) {
        const V4 pa = load_v4(node_soa, a, m, i);
        for (int b = a + 1; b < n_ext; ++b) {
            const double d = mass2(pa + load_v4(node_soa, b, m, i)) - m2;
            const double bw = 1.0 / (d * d + mw2);
            sum += bw;
            if (bw > big1) {
                big2 = big1;
                big1 = bw;
            } else if (bw > big2) {
                big2 = bw;
            }
        }
    }
    const V4 p0 = load_v4(node_soa, 0, m, i);
    double tprod = 1;
    for (int b = 2; b < n_ext; ++b) tprod *= 1.0 / (fabs(mass2(p0 + load_v4(node_soa, b, m, i))) + mt2);
    return (top2 ? big1 * big2 : sum) * tprod;
}

// Every channel's densities: channel c's at tile point i is
// p[c * stride + i] (the per-record array of an iteration from the tile's
// first record on, or a tile's own buffer).
struct Densities {
    double *p;
    long long stride;
};

// 1 / sum_c alpha_c / dens_c / vw_c at tile point i in channel order
// (Integrand.hh:118-122).  Eight channels' values are in flight before the
// first division: one at a time, the divisions' slow-path branches kept the
// next loads back (0.151 against 0.097 ms per 1e6 points of 15 channels).
// dens_row: the point's densities in channel order, where asked for.
__device__ __forceinline__ double pp_weight_sum(int nch, const double *__restrict__ alpha, Densities dens,
                                                const double *__restrict__ vwv, long long m, long long i,
                                                double *__restrict__ dens_row = nullptr) {
    const double *dp = dens.p + i, *vp = vwv + i;
    double acc = 0.0;
    for (int c0 = 0; c0 < nch; c0 += 8) {
        double d[8], v[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const int c = min(c0 + k, nch - 1);
            d[k] = __ldg(dp + c * dens.stride);
            v[k] = __ldg(vp + c * m);
        }
#pragma unroll
        for (int k = 0; k < 8; ++k)
            if (c0 + k < nch) {
                acc += __ldg(alpha + c0 + k) / d[k] / v[k];
                if (dens_row) dens_row[c0 + k] = d[k];
            }
    }
    return 1.0 / acc;
}

__device__ __forceinline__ void pp_combine_point(const PointProgram *__restrict__ pp, const double *__restrict__ alpha,
                                                 Densities dens, const double *__restrict__ vwv,
                                                 const double *__restrict__ node_soa, long long m, long long i,
                                                 long long r, const IntegrandDesc *__restrict__ f,
                                                 double *__restrict__ rec_val, double *__restrict__ rec_wgt,
                                                 uint8_t *__restrict__ rec_ok) {
    double wgt = pp_weight_sum(pp->nch, alpha, dens, vwv, m, i);
    const double fv = eval_momenta_soa(f, node_soa, m, i, pp->n_ext);
    double val = wgt == 0 ? 0 : fv * wgt;
    uint8_t ok = 1;
    if (isnan(val)) {
        val = wgt = 0;
        ok = 0;
    }
    rec_val[r] = val;
    rec_wgt[r] = wgt;
    rec_ok[r] = ok;
}

// The grid set's search tables (grid.cuh), every channel's rows back to back.
struct GridTables {
    const double *edges;      // [nch][dims][bins + 1]
    const uint32_t *entries;  // [nch][dims][grid_cells(bins)]
    const double *ws;         // [nch][dims][width_row(bins)]
};

// Shared-memory bytes of the channel step: the position and factor rows, and
// one channel's tables where they are staged.
constexpr int kMaxFactors = 2 * CHILI_MAX_DECAYS + 1;
__host__ __device__ inline size_t channel_smem_bytes(int dims, int bins, bool tables) {
    const size_t rows = 16 * ((sizeof(int32_t) * (2 * static_cast<size_t>(dims) + kMaxFactors) + 15) / 16);
    return rows + (tables ? static_cast<size_t>(dims) * (4 * static_cast<size_t>(grid_cells(bins)) + 8 * width_row(bins)) : 0);
}

// Dynamic shared memory that kernels with tables of the grid's size may take.
constexpr size_t kMaxDynSmem = 200 * 1024;

// Launch shape of the channel step: one channel's tables in shared memory
// where they fit, and as many threads per block as keep 32 warps on an SM
// beside them.
constexpr int channel_max_threads(int dims) { return dims > 10 && dims <= 16 ? 1024 : 512; }
struct ChannelShape {
    bool tables;
    size_t smem;
    int threads;
};
inline ChannelShape channel_shape(int dims, int bins, bool want_tables) {
    const bool tab = want_tables && channel_smem_bytes(dims, bins, true) <= kMaxDynSmem;
    const size_t smem = channel_smem_bytes(dims, bins, tab);
    return {tab, smem, !tab || smem <= 54 * 1024 ? 256 : (smem <= 110 * 1024 ? 512 : channel_max_threads(dims))};
}
// The same for the grouped launches of batched tasks, whose blocks take a
// couple of thousand points: tables that leave no room for 32 warps are read
// from global memory (14 tasks of 10 dimensions at 300 bins, 196 KB: 2.54 ms an
// iteration staged, 2.32 read from there; 200 bins, 98 KB: 2.10 against 2.15; 11
// tasks of 13 dimensions at 200 bins, 127 KB and 32 warps: 1.32 against 1.35).
inline ChannelShape grouped_channel_shape(int dims, int bins, bool want_tables) {
    const ChannelShape s = channel_shape(dims, bins, want_tables);
    return s.smem > 110 * 1024 && s.threads < 1024 ? channel_shape(dims, bins, false) : s;
}

// 16 bytes from global to shared memory (both 16-byte aligned), and the wait
// for this thread's copies.
__device__ __forceinline__ void copy16_async(uint32_t dst, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void copy_async_wait() {
    asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
}

// The channel step of one block: channel c's density (the product of its
// items in the reference's order, Channel.cc:40-61) and its VEGAS weight at
// the tile points [i0, i1) on the uniforms that the position map selects, the
// density and, for the point's own channel, its bins record (REC: own_out is
// uint4 rows, mc_device.cuh) or its uniforms (own_out, [point][DIMS], may be
// null).  When c's
// chain fails, its last uniform is the one the shared buffer still holds: the
// last uniform of the latest earlier channel whose chain did not fail (zero
// if none).  TAB: channel c's entries and widths are staged in shared memory
// first; the edges, which only undecided searches read, stay in global
// memory.  Three passes over the dimensions: the uniforms are loaded, then
// counted without a branch (the undecided ones noted in a mask and searched
// afterwards: 0.7% of them on trained 200-bin grids, but some lane of a warp
// in every fifth search), then the widths multiplied in the reference's
// order.  smem: channel_smem_bytes.
template <int DIMS, bool TAB, int F, bool REC>
__device__ __forceinline__ void pp_channel_block(const PointProgram *__restrict__ pp, const GridTables &T, int bins,
                                                 const double *__restrict__ memo, const uint8_t *__restrict__ cfail,
                                                 const int32_t *__restrict__ ich_tile, long long m, Densities dens,
                                                 double *__restrict__ vwv, void *__restrict__ own_out, long long base,
                                                 long long i0, long long i1, int c, void *smem) {
    const int cells = grid_cells(bins);
    const double scale = static_cast<double>(cells) * static_cast<double>(1 << F);
    int32_t *pos_s = static_cast<int32_t *>(smem);  // [2][DIMS]: chain found, chain failed
    uint32_t *en_s = reinterpret_cast<uint32_t *>(static_cast<char *>(smem) + channel_smem_bytes(DIMS, bins, false));
    double *ws_s = reinterpret_cast<double *>(en_s + static_cast<size_t>(DIMS) * cells);
    const PPChannel &C = pp->ch[c];
    const double *g = T.edges + static_cast<size_t>(c) * DIMS * (bins + 1);
    const uint32_t *en = T.entries + static_cast<size_t>(c) * DIMS * cells;
    const int wn = width_row(bins);
    const double *ws = T.ws + static_cast<size_t>(c) * DIMS * wn;
    for (int p = threadIdx.x; p < 2 * DIMS; p += blockDim.x)
        pos_s[p] = p < DIMS ? pp->pos_src[c][p] : pp->pos_src_fail[c][p - DIMS];
    // the density's factors: decay propagators, two-body decays, the chain
    const int n_dec = C.n_dec, n_fac = n_dec + C.n_sd, chain = C.chain;
    int32_t *fac_s = pos_s + 2 * DIMS;
    for (int k = threadIdx.x; k <= n_fac; k += blockDim.x)
        fac_s[k] = k < n_dec ? pp->memo_dw + 2 * C.dw[k]
                             : (k < n_fac ? pp->memo_sw + 3 * C.sw[k - n_dec] : pp->memo_chain + 2 * chain);
    if constexpr (TAB) {
        // all copies in flight at once (rows are multiples of 16 bytes): a
        // loop of loads and stores took one memory latency per pass of the block
        const char *src = reinterpret_cast<const char *>(en), *srcw = reinterpret_cast<const char *>(ws);
        const uint32_t dst = static_cast<uint32_t>(__cvta_generic_to_shared(en_s));
        const uint32_t dstw = static_cast<uint32_t>(__cvta_generic_to_shared(ws_s));
        for (int k = threadIdx.x; k < DIMS * (cells >> 2); k += blockDim.x) copy16_async(dst + 16 * k, src + 16 * k);
        for (int k = threadIdx.x; k < DIMS * (wn >> 1); k += blockDim.x) copy16_async(dstw + 16 * k, srcw + 16 * k);
        copy_async_wait();
        en = en_s;
        ws = ws_s;
    }
    __syncthreads();
    const long long ms = m;
    double *dens_c = dens.p + c * dens.stride, *vw_c = vwv + c * ms;
    const uint8_t *fail_c = cfail + chain * ms;
    const unsigned row_bytes = static_cast<unsigned>(m) * 8u;  // tiles stay below 2^28 points
    constexpr int NW = 4 * ((DIMS + 8) / 8);                   // words of a bins record
    constexpr int kFacAhead = 2;
    uint8_t fail_next = i0 + threadIdx.x < i1 ? fail_c[i0 + threadIdx.x] : 0;
#pragma unroll 1
    for (long long i = i0 + threadIdx.x; i < i1; i += blockDim.x) {
        const char *mi = reinterpret_cast<const char *>(memo + i);
        auto at = [&](int slot) {  // memo slot of point i
            return *reinterpret_cast<const double *>(mi + static_cast<unsigned long long>(row_bytes) *
                                                              static_cast<unsigned>(slot));
        };
        const bool fail = fail_next != 0;
        if (i + blockDim.x < i1) fail_next = fail_c[i + blockDim.x];
        const int32_t *pos = pos_s + (fail ? DIMS : 0);
        double x[DIMS];
#pragma unroll
        for (int p = 0; p < DIMS - 1; ++p) x[p] = at(pos[p]);
        if (!fail) {
            x[DIMS - 1] = at(pos[DIMS - 1]);
        } else {
            double stale = 0.0;
            for (int k = c - 1; k >= 0; --k) {
                if (!cfail[pp->ch[k].chain * ms + i]) {
                    stale = at(pp->pos_src[k][DIMS - 1]);
                    break;
                }
            }
            x[DIMS - 1] = stale;
        }
        // the first factors loaded together, before the first product waits
        const double wt = at(fac_s[n_fac]);
        double fv[kFacAhead], wdec = 1, sw = 1;
        // WgtDecays divides the running product by 2 pi after every decay (Channel.cc:107-111)
        auto decay = [&](double w) { wdec = div_by(wdec * w, kTwoPi, kRcpTwoPi); };
#pragma unroll
        for (int k = 0; k < kFacAhead; ++k) fv[k] = at(fac_s[min(k, n_fac)]);
        const bool own = (REC || own_out) && ich_tile[i] == c;
        if (!REC && own) {
            double *o = static_cast<double *>(own_out) + (base + i) * DIMS;
#pragma unroll
            for (int p = 0; p < DIMS; ++p) o[p] = x[p];
        }
        uint32_t rec[NW], todo = 0;
#pragma unroll
        for (int k = 0; k < NW; ++k) rec[k] = 0;
#pragma unroll
        for (int p = 0; p < DIMS; ++p) {
            bool slow;
            const int n = cell_count<!TAB, F>(en + p * cells, cells, scale, x[p], slow);
            if (slow) todo |= 1u << p;
            else rec[p >> 1] |= static_cast<uint32_t>(n) << (16 * (p & 1) + 3);
        }
        while (todo) {
            const int p = __ffs(todo) - 1;
            todo &= todo - 1;
            double v = x[DIMS - 1];
            if (p < DIMS - 1) v = at(pos[p]);
            const uint32_t n = static_cast<uint32_t>(cell_count_slow<!TAB, F>(g + p * (bins + 1), en + p * cells, bins,
                                                                              cells, scale, v))
                               << (16 * (p & 1) + 3);
#pragma unroll
            for (int k = 0; k < (DIMS + 1) / 2; ++k)  // masks, not an index: rec stays in registers
                rec[k] |= n & (0u - static_cast<uint32_t>(k == (p >> 1)));
        }
        // behind the searches, where the uniforms' registers are free (before
        // them the products spilled: 2->6 1.85 instead of 1.57 ms)
#pragma unroll
        for (int k = 0; k < kFacAhead; ++k) {
            if (k < n_dec) decay(fv[k]);
            else if (k < n_fac) sw *= fv[k];
        }
        for (int k = kFacAhead; k < n_fac; ++k) {
            if (k < n_dec) decay(at(fac_s[k]));
            else sw *= at(fac_s[k]);
        }
        const double dc = wdec * wt * sw;
        double vw = 1.0;
#pragma unroll
        for (int p = 0; p < DIMS; ++p) {
            const uint32_t off = (rec[p >> 1] >> (16 * (p & 1))) & 0xffffu;
            vw = __dmul_rn(vw, tab_ld<!TAB>(reinterpret_cast<const double *>(
                                   reinterpret_cast<const char *>(ws + p * wn) + off)));
        }
        dens_c[i] = dc;
        vw_c[i] = vw;
        if (REC && own) {
            rec[DIMS >> 1] |= static_cast<uint32_t>(c) << (16 * (DIMS & 1));
            uint4 *o = static_cast<uint4 *>(own_out) + (base + i) * (NW / 4);
#pragma unroll
            for (int k = 0; k < NW / 4; ++k) o[k] = make_uint4(rec[4 * k], rec[4 * k + 1], rec[4 * k + 2], rec[4 * k + 3]);
        }
    }
}

// (The body as a device function, so that a grouped launch can run it for
// one piece of work per block.)
__device__ __forceinline__ void mc_scan_body(const int32_t *__restrict__ block_count, int nb,
                                             const uint8_t *__restrict__ flag, long long m, long long needed,
                                             const long long *__restrict__ remaining, int cut_at_remaining,
                                             long long *__restrict__ block_off, RoundCtl *__restrict__ ctl) {
    if (remaining) {
        const long long rem = *remaining;
        if (rem <= 0) {
            if (threadIdx.x == 0) {
                ctl->cut = 0;
                ctl->n_acc = 0;
            }
            return;
        }
        if (cut_at_remaining) needed = rem;
    }
    __shared__ long long wsum[32];
    __shared__ long long running_s;
    __shared__ int cut_block_s;
    __shared__ long long cut_off_s;
    if (threadIdx.x == 0) {
        running_s = 0;
        cut_block_s = -1;
        cut_off_s = 0;
    }
    __syncthreads();
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int base = 0; base < nb; base += 1024) {
        const int i = base + threadIdx.x;
        const long long c = i < nb ? block_count[i] : 0;
        long long incl = c;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const long long t = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += t;
        }
        if (lane == 31) wsum[w] = incl;
        __syncthreads();
        if (w == 0) {
            long long v = wsum[lane];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const long long t = __shfl_up_sync(0xffffffffu, v, o);
                if (lane >= o) v += t;
            }
            wsum[lane] = v;  // inclusive warp totals
        }
        __syncthreads();
        const long long warp_excl = w > 0 ? wsum[w - 1] : 0;
        const long long off = running_s + warp_excl + incl - c;
        if (i < nb) {
            block_off[i] = off;
            if (off < needed && needed <= off + c) {
                cut_block_s = i;
                cut_off_s = off;
            }
        }
        __syncthreads();
        if (threadIdx.x == 0) running_s += wsum[31];
        __syncthreads();
    }
    const long long total = running_s;
    if (cut_block_s < 0) {
        if (threadIdx.x == 0) {
            ctl->cut = m;
            ctl->n_acc = total;
        }
        return;
    }
    // position of the r-th accepted point inside the cut block
    const long long r = needed - cut_off_s;
    const long long k = static_cast<long long>(cut_block_s) * kFwdBlock + threadIdx.x;
    int f = 0;
    if (threadIdx.x < kFwdBlock && k < m) f = flag[k] ? 1 : 0;
    long long incl = f;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const long long t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
    }
    __syncthreads();
    if (lane == 31) wsum[w] = incl;
    __syncthreads();
    long long pre = 0;
    for (int q = 0; q < w; ++q) pre += wsum[q];
    incl += pre;
    if (threadIdx.x < kFwdBlock && f && incl == r) {
        ctl->cut = k + 1;
        ctl->n_acc = needed;
    }
}

// Block bx of the ordered compaction of the accepted points.
__device__ __forceinline__ void mc_compact_block(const uint8_t *__restrict__ flag,
                                                 const long long *__restrict__ block_off,
                                                 const RoundCtl *__restrict__ ctl, long long m,
                                                 int32_t *__restrict__ list, long long bx) {
    const long long k = bx * static_cast<long long>(kFwdBlock) + threadIdx.x;
    const long long cut = ctl->cut;
    const int a = (k < m && k < cut) ? flag[k] : 0;
    const unsigned ballot = __ballot_sync(0xffffffffu, a);
    __shared__ int wc[kFwdBlock / 32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (lane == 0) wc[w] = __popc(ballot);
    __syncthreads();
    int pre = 0;
    for (int q = 0; q < w; ++q) pre += wc[q];
    if (a) {
        const long long pos = block_off[bx] + pre + __popc(ballot & ((1u << lane) - 1u));
        list[pos] = static_cast<int32_t>(k);
    }
}

}  // namespace chili_dev
