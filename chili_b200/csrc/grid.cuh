// grid.cuh -- device form of chili::AdaptiveMap (VEGAS grid).
//
// A grid set holds nch grids of `dims` x (bins+1) edges, each grid in the
// reference layout edges[dim*(bins+1) + k] (AdaptiveMap.hh:29-40), grids back
// to back.  The forward map and the bin search use explicitly rounded
// multiply/add so that x, J and bin indices are bit-identical to the
// reference's (compiled without FMA contraction) for identical inputs.
#pragma once

#include "chili_gpu.h"
#include "common.cuh"

namespace chili_dev {

// Table reads: through the read-only path (global tables, NC = true) or
// plain loads (tables staged in shared memory, NC = false).
template <bool NC, class T>
__device__ __forceinline__ T tab_ld(const T *p) {
    if constexpr (NC) return __ldg(p);
    else return *p;
}

// std::lower_bound over edges[0..bins) with libstdc++'s probe sequence, then
// "- 1" as in AdaptiveMap::FindBin (AdaptiveMap.cc:34-38).  Returns -1 where
// the reference returns SIZE_MAX (x <= edges[0] or x NaN).
template <bool NC = true>
__device__ __forceinline__ int find_bin(const double *__restrict__ e, int bins, double x) {
    int first = 0, len = bins;
    while (len > 0) {
        const int half = len >> 1;
        const int mid = first + half;
        if (tab_ld<NC>(e + mid) < x) {
            first = mid + 1;
            len = len - half - 1;
        } else {
            len = half;
        }
    }
    return first - 1;
}

// The 8 bytes before the reference's edge table.  AdaptiveMap::width(0,
// SIZE_MAX) reads m_hist[-1]; under glibc malloc that is the size word of the
// vector's heap chunk: (8*dims*(bins+1) + 8) rounded up to 16, with the
// PREV_INUSE bit set (mmapped chunks, from 128 KiB up, round to pages and set
// IS_MMAPPED).  As a double it is a positive denormal; whether a channel's
// term then overflows to -inf or stays finite depends on its exact value, so
// the host computes it per grid shape (edge_before_table()).
__host__ __device__ inline double edge_before_table(int dims, int bins) {
    const unsigned long long req = 8ull * static_cast<unsigned long long>(dims) * (bins + 1);
    unsigned long long word;
    if (req + 8 >= 128ull * 1024) word = ((req + 16 + 4095) & ~4095ull) | 2ull;
    else {
        word = (req + 8 + 15) & ~15ull;
        word = (word < 32ull ? 32ull : word) | 1ull;
    }
    union {
        unsigned long long u;
        double d;
    } cv;
    cv.u = word;
    return cv.d;
}

// width(dim, bin) of the flat edge table, including the reference's reading
// of bin == SIZE_MAX: lower_edge at flat index dim*(bins+1) - 1 (the previous
// dimension's last edge, or the word before the table for dim 0).
template <bool NC = true>
__device__ __forceinline__ double bin_width(const double *__restrict__ g, int bins, int dim, int bin,
                                            double before) {
    const int base = dim * (bins + 1);
    if (bin >= 0) return __dsub_rn(tab_ld<NC>(g + base + bin + 1), tab_ld<NC>(g + base + bin));
    const double lower = dim > 0 ? tab_ld<NC>(g + base - 1) : before;
    return __dsub_rn(tab_ld<NC>(g + base), lower);
}

// AdaptiveMap::operator() (AdaptiveMap.cc:40-56) on one point: x in place,
// returns the Jacobian.
__device__ __forceinline__ double grid_map(const double *__restrict__ g, int dims, int bins, double *x) {
    double jac = 1.0;
    const double fb = static_cast<double>(bins);
    for (int d = 0; d < dims; ++d) {
        const double pos = __dmul_rn(x[d], fb);
        const int idx = static_cast<int>(pos);
        const double loc = __dsub_rn(pos, static_cast<double>(idx));
        const double *e = g + d * (bins + 1);
        const double left = __ldg(e + idx);
        const double size = __dsub_rn(__ldg(e + idx + 1), left);
        x[d] = __dadd_rn(left, __dmul_rn(loc, size));
        jac = __dmul_rn(jac, __dmul_rn(size, fb));
    }
    return jac;
}

// AdaptiveMap::GenerateWeight (AdaptiveMap.cc:58-65).
__device__ __forceinline__ double grid_weight(const double *__restrict__ g, int dims, int bins,
                                              const double *x, double before) {
    double jac = 1.0;
    const double fb = static_cast<double>(bins);
    for (int d = 0; d < dims; ++d) {
        const int b = find_bin(g + d * (bins + 1), bins, x[d]);
        jac = __dmul_rn(jac, __dmul_rn(bin_width(g, bins, d, b, before), fb));
    }
    return jac;
}

// Flat histogram slot of dimension d's bin b the way Integrand::AddTrainData
// and Vegas::operator() index it (train[d*bins + FindBin]); a FindBin of
// SIZE_MAX wraps to d*bins - 1, which for d == 0 lies before the histogram:
// that slot is reported as -1 (skipped).
__device__ __forceinline__ int train_slot(int d, int bins, int b) {
    const int s = d * bins + b;
    return s;  // b == -1 and d == 0 gives -1
}

// ------------------------------------------------------------ cell search
// FindBin through a table of H uniform cells over [0, 1), H a power of two.
// Every coordinate v in [0, 1) has an integer image g(v) = floor(v H 2^F),
// exact and monotone: one round-down multiply-add onto 2^52 leaves it in the
// low word.  Its upper bits are the cell, its lower F bits the place in the
// cell.  A cell's entry packs the number of edges e[k], k < bins, in lower
// cells and the places f1 <= f2 of the cell's first two edges, so that one
// multiply-add counts the edges below x:
//   entry   = start << (2F+2) | (2^(F+1) - 1 - f1) << (F+1) | (2^F - 1 - f2)
//   entry + f (2^(F+1) + 1): f > f1 carries into start, f > f2 sets bit F
// (an absent edge's field is 0).  g(x) > g(e) implies x > e and g(x) < g(e)
// implies x < e, so the count is FindBin + 1.  A field of ones in the sum is
// an equal place (2^-F of the points); bit F set in the entry marks a cell
// with more than two edges; both compare the cell's edges themselves
// (cell_count_slow).  x outside [0, 1) and rows that are not monotone inside [0, 1)
// (every entry start all ones, bit F) take the plain search.  The bins are
// those of find_bin in every case.
//
// Why: a hint of two cells per bin and a binary search on the edges took 96
// issued instructions and 16 shared-memory wavefronts per search and bound
// the channel step by issue; this search is one 4-byte and (for the width)
// one 8-byte table read.  8 cells per bin: on trained 100-bin grids 1% of a
// grid's own points fall in a cell with more than two edges (4 per bin: 4%).
constexpr int kMaxCells = 4096;

__host__ __device__ inline int grid_cells(int bins) {
    int h = 64;
    while (h < 8 * bins && h < kMaxCells) h <<= 1;
    return h;
}

// Place bits: 11 where the count and the marker fit the remaining 8 bits, else
// 8 (14 bits).
__host__ __device__ constexpr int cell_fbits(int bins) { return bins <= 254 ? 11 : 8; }

// FindBin + 1 of x from the row's entries (TABLE_NC: in global memory, else
// staged in shared memory), cells = grid_cells(bins), scale = cells 2^F;
// slow: the entry does not decide, and the count is find_bin's.
template <bool TABLE_NC, int F>
__device__ __forceinline__ int cell_count(const uint32_t *__restrict__ entries, int cells, double scale, double x,
                                          bool &slow) {
    const double t = __fma_rd(x, scale, 0x1p52);
    const uint32_t lo = static_cast<uint32_t>(__double2loint(t));
    const uint32_t q = tab_ld<TABLE_NC>(entries + ((lo >> F) & (cells - 1)));
    const uint32_t s = q + (lo & ((1u << F) - 1u)) * ((2u << F) + 1u);
    const uint32_t inv = ~s;
    slow = __double2hiint(t) != 0x43300000 || lo >= (static_cast<uint32_t>(cells) << F) || (q & (1u << F)) != 0 ||
           (inv & ((1u << F) - 1u)) == 0 || (inv & (((2u << F) - 1u) << (F + 1))) == 0;
    return static_cast<int>(s >> (2 * F + 2)) + static_cast<int>((s >> F) & 1u);
}

// FindBin + 1 where the entry does not decide, on the row of edges e (global
// memory): among the cell's edges, three at the quarters at a time, the last
// four together.  (A trained peak puts most edges, and most points, into few
// cells: read from the cell's first edge on, 1e7 searches among 1000 edges in one
// cell took 2.7 ms, so 0.17; the channel step of 1e5 trained 2->4 points at 1000
// bins 0.44 -> 0.11 ms.)
template <bool TABLE_NC, int F>
__device__ __forceinline__ int cell_count_slow(const double *__restrict__ e, const uint32_t *__restrict__ entries,
                                               int bins, int cells, double scale, double x) {
    // outside [0, 1) (points outside a channel's region, uncut events): any
    // cell tells whether the row is monotone inside it
    const bool in = x >= 0.0 && x < 1.0;
    const uint32_t lo = in ? static_cast<uint32_t>(__double2loint(__fma_rd(x, scale, 0x1p52))) : 0u;
    const int cell = static_cast<int>((lo >> F) & (cells - 1));
    int k = static_cast<int>(tab_ld<TABLE_NC>(entries + cell) >> (2 * F + 2));
    if (k == static_cast<int>(0xffffffffu >> (2 * F + 2))) return find_bin<true>(e, bins, x) + 1;
    if (!in) return x >= 1.0 ? bins : 0;
    // the count lies between this cell's start and the next one's
    int len = (cell + 1 < cells ? static_cast<int>(tab_ld<TABLE_NC>(entries + cell + 1) >> (2 * F + 2)) : bins) - k;
    while (len > 4) {
        const int s = len >> 2;
        const int n = (__ldg(e + k + s) < x) + (__ldg(e + k + 2 * s) < x) + (__ldg(e + k + 3 * s) < x);
        k += n > 0 ? n * s + 1 : 0;
        len = n == 0 ? s : (n < 3 ? s - 1 : len - 3 * s - 1);
    }
    int n = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) n += (j < len && __ldg(e + min(k + j, bins)) < x) ? 1 : 0;
    return k + n;
}

// Doubles of a row of scaled widths: bins + 1, rounded to 16 bytes.
__host__ __device__ inline int width_row(int bins) { return (bins + 2) & ~1; }

// The entries of row (dimension) dim of the grid g (dims x (bins+1) edges)
// and its scaled widths: ws[0] the reference's reading of bin == SIZE_MAX,
// ws[1 + k] = (e[k+1] - e[k]) * bins (the factors of
// AdaptiveMap::GenerateWeight, rounded as there).  Built by one block.
__device__ __forceinline__ void build_cell_row(const double *__restrict__ g, int dims, int bins, int dim,
                                               uint32_t *__restrict__ entries, double *__restrict__ ws) {
    __shared__ uint32_t g_s[CHILI_MAX_BINS];
    const double *e = g + static_cast<size_t>(dim) * (bins + 1);
    const int F = cell_fbits(bins), cells = grid_cells(bins);
    const double scale = static_cast<double>(cells) * static_cast<double>(1 << F), fb = static_cast<double>(bins);
    const uint32_t mask = (1u << F) - 1u;
    int bad = 0;
    for (int k = threadIdx.x; k < bins; k += blockDim.x) {
        const double a = e[k];
        if (!(a >= 0.0 && a < 1.0) || (k + 1 < bins && !(a <= e[k + 1]))) bad = 1;
        g_s[k] = static_cast<uint32_t>(__double2loint(__fma_rd(a, scale, 0x1p52)));
        ws[1 + k] = __dmul_rn(__dsub_rn(e[k + 1], a), fb);
    }
    if (threadIdx.x == 0) ws[0] = __dmul_rn(bin_width<false>(g, bins, dim, -1, edge_before_table(dims, bins)), fb);
    bad = __syncthreads_or(bad);
    for (int j = threadIdx.x; j < cells; j += blockDim.x) {
        if (bad) {
            entries[j] = (0xffffffffu << (2 * F + 2)) | 1u << F;
            continue;
        }
        int first = 0, len = bins;  // edges in lower cells
        while (len > 0) {
            const int half = len >> 1, mid = first + half;
            if (static_cast<int>(g_s[mid] >> F) < j) {
                first = mid + 1;
                len = len - half - 1;
            } else {
                len = half;
            }
        }
        int in = 0;
        while (in < 3 && first + in < bins && static_cast<int>(g_s[first + in] >> F) == j) ++in;
        uint32_t q = static_cast<uint32_t>(first) << (2 * F + 2);
        if (in > 0) q |= (2u * mask + 1u - (g_s[first] & mask)) << (F + 1);
        if (in > 1) q |= mask - (g_s[first + 1] & mask);
        if (in > 2) q = (static_cast<uint32_t>(first) << (2 * F + 2)) | 1u << F;
        entries[j] = q;
    }
    __syncthreads();  // g_s is free for another row
}

}  // namespace chili_dev
