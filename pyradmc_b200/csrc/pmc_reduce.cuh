// pmc_reduce.cuh — batch fold, finalize and Dij truncation/compaction.
//
// These are HBM-streaming kernels over the [columns][voxels] maps; the
// engine's fold, finalize and truncation visit only the 32-byte sectors that
// deposits touched (sector bitmaps below).  Every
// float64 operation is written with an explicit round-to-nearest intrinsic, so
// nothing is contracted into an FMA: the results equal, bit for bit, the numpy
// scorers they restate —
//   fold      BatchedBeamletScorer.end_batch   scoring/dij.py:155-174
//             (BatchedDoseScorer.end_batch     scoring/dose.py:169-186)
//   finalize  BatchedBeamletScorer.finalize    scoring/dij.py:176-191
//   truncate  DijAssembler.add_block           scoring/dij.py:351-366
// The compaction's prefix sum runs on the device (the Warp engine read the
// per-chunk counts back and scanned them with numpy, engine.py:1517-1525).
#pragma once

#include "pmc_common.cuh"
#include "pmc_scan.cuh"

namespace pmc {

constexpr int kReduceThreads = 256;
constexpr int kTileVoxels = 4096;  // truncation tile: one block per (column, tile)

__device__ __forceinline__ unsigned long long warp_sum_u64(unsigned long long v) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    return v;
}

__device__ __forceinline__ bool keep_entry(double m, double threshold) {
    return m >= threshold && m > 0.0;
}

// ---- sector bitmaps ----------------------------------------------------------------
// The engine's dense maps (int64 quanta, float64 sums) are laid out
// [column][stride] with the column stride a multiple of kTileVoxels, so that
// entry e of the map belongs to the 32-byte sector e >> 2 and to bit
// (e >> 2) & 31 of bitmap word e >> 7 (128 entries per word, 32 words per
// truncation tile).  Every atomic deposit also ORs its sector's bit into the
// `dirty` bitmap; the fold visits only dirty sectors, clears their bits and
// records them in the `touched` bitmap (every sector any batch ever scored).
// The sums of a Dij are never cleared in bulk: a sector's first fold writes all
// four of its entries (d or +0.0), and finalize / truncation read touched
// sectors only.  0.0 + d == d, so a first write equals the reference's s += d.
constexpr int kSectorEntries = 4;
constexpr int kWordEntries = 128;
static_assert(kTileVoxels == 32 * kWordEntries, "one bitmap word per lane of a tile's warp");

__device__ __forceinline__ void mark_dirty(unsigned int* dirty, long long flat) {
    atomicOr(dirty + (flat >> 7), 1u << ((unsigned)(flat >> 2) & 31u));
}

// Position of set bit number n (from 0) of w; some position for n >= popc(w).
// Five popcounts: the library's __fns is a loop over the bits.
__device__ __forceinline__ int nth_set_bit(unsigned int w, int n) {
    int pos = 0;
#pragma unroll
    for (int step = 16; step >= 1; step >>= 1) {
        const int below = __popc((w >> pos) & ((1u << step) - 1u));
        if (below <= n) {
            n -= below;
            pos += step;
        }
    }
    return pos & 31;
}

// One warp holds the 32 bitmap words of a tile (word j in lane j); lane order
// then bit order is ascending sector order.  `incl` is the warp's inclusive
// scan of the words' popcounts.  Returns the lane whose word holds set bit
// number k (of the whole tile) and that bit's position; every lane must call
// it (it shuffles), and the result is meaningless for k >= the tile's total.
__device__ __forceinline__ int nth_set_sector(unsigned int w, int incl, int k, int& bit) {
    int j = 0;
#pragma unroll
    for (int step = 16; step >= 1; step >>= 1) {
        const int v = __shfl_sync(0xffffffffu, incl, j + step - 1);
        if (v <= k) j += step;
    }
    const unsigned int wj = __shfl_sync(0xffffffffu, w, j);
    const int before = __shfl_sync(0xffffffffu, incl, j) - __popc(wj);
    bit = nth_set_bit(wj, k - before);
    return j;
}

__device__ __forceinline__ int warp_inclusive_scan(int v) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, v, off);
        if (lane >= off) v += y;
    }
    return v;
}

// The four entries of one sector as two 16-byte halves (sectors are 32-byte
// aligned: the column stride is a multiple of kTileVoxels).
struct SectorD {
    double v[kSectorEntries];
    __device__ __forceinline__ void load(const double* p) {
        const double2 lo = reinterpret_cast<const double2*>(p)[0], hi = reinterpret_cast<const double2*>(p)[1];
        v[0] = lo.x; v[1] = lo.y; v[2] = hi.x; v[3] = hi.y;
    }
    __device__ __forceinline__ void store(double* p) const {
        reinterpret_cast<double2*>(p)[0] = make_double2(v[0], v[1]);
        reinterpret_cast<double2*>(p)[1] = make_double2(v[2], v[3]);
    }
};

// mean = S1/n, sigma = sqrt(max(0, S2/n - mean^2) * n / (n - 1) / n) of one entry, in place.
__device__ __forceinline__ void finalize_entry(double& x, double& y, double n, int n_batches) {
    if (x == 0.0 && y == 0.0) return;  // mean and sigma are already +0.0
    const double mean = __ddiv_rn(x, n);
    double sigma = 0.0;
    if (n_batches > 1) {
        double var = __dsub_rn(__ddiv_rn(y, n), __dmul_rn(mean, mean));
        var = var > 0.0 ? var : 0.0;
        var = __ddiv_rn(__dmul_rn(var, n), n - 1.0);
        sigma = __dsqrt_rn(__ddiv_rn(var, n));
    }
    x = mean;
    y = sigma;
}

// The largest bit pattern of a column's means, which is the largest mean while none is
// negative.  A deposit of a slightly negative float32 energy (about -1e-9 MeV) that meets
// no other in its voxel leaves a negative mean: its sign bit makes it the maximum, the
// column's threshold is negative and all its positive entries are kept (5 of 40 columns
// at 2e5 histories each on the 128^3 phantom).  The reference takes the largest value;
// colmax_kernel, which reads finished means, does too.
__device__ __forceinline__ void column_max(unsigned long long best, unsigned long long* col_max_bits) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        const unsigned long long o = __shfl_xor_sync(0xffffffffu, best, off);
        best = o > best ? o : best;
    }
    if ((threadIdx.x & 31) == 0 && best) atomicMax(col_max_bits, best);
}

// How the fold and finalize walk the sector bitmaps.  A part is `words` consecutive
// words (1 to 32, dividing a tile's 32) of one column, one per lane of a warp.  The
// warps of a resident grid claim `claim` parts at a time from a counter, the next
// part's words on their way while the current one is folded.  Most parts of a Dij
// are empty and the full ones lie side by side (a beam's core): with a warp
// launched per tile, the launches of the empty ones and the blocks that held one
// full tile each took most of the time (16 % of the warps active), and parts dealt
// out in turn still left some warps half again as long as the others.
struct FoldShape {
    long long n_vox, stride;  // voxels and entries of a column
    int words;                // bitmap words per part
    int parts_per_col;
    unsigned int n_parts, claim;
    unsigned int* next;       // parts claimed so far (zero at launch)
    int n_maps;               // quanta maps of the wave, in batch order
    long long map_entries;    // entries of one map
};

// The next claim of a warp: its first part (n_parts and up: none left).
__device__ __forceinline__ unsigned int claim_parts(const FoldShape& f) {
    unsigned int t = 0u;
    if ((threadIdx.x & 31) == 0) t = atomicAdd(f.next, f.claim);
    return __shfl_sync(0xffffffffu, t, 0);
}

// x / y correctly rounded, from r = 1 / y correctly rounded: two Newton corrections
// of x r, each with an exact remainder (Markstein, "Computation of elementary
// functions on the IBM RISC System/6000 processor", IBM J. Res. Dev. 34, 1990: the
// second one rounds correctly, the first having left a quotient within one unit in
// the last place).  For y = r = 0 it gives 0; else y must be a usual divisor: with
// dividends of 0 or 1e-9 to 1e10 no step then overflows or loses bits.
__device__ __forceinline__ bool usual_divisor(double y) { return y >= 0x1p-900 && y <= 0x1p900; }
__device__ __forceinline__ double divide_by(double x, double y, double r) {
    double q = __dmul_rn(x, r);
    q = __fma_rn(__fma_rn(-q, y, x), r, q);
    return __fma_rn(__fma_rn(-q, y, x), r, q);
}

// *odd = 1 where some mass times a count of histories (1 to 2^100) is no usual divisor
// (no mass at all is none that the fold divides by).
__global__ void odd_masses_kernel(const double* __restrict__ mass, long long n, unsigned int* odd) {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x) {
        const double m = mass[i];
        if (m > 0.0 && !(usual_divisor(m) && usual_divisor(m * 0x1p100))) *odd = 1u;
    }
}

// Fold a wave's quanta maps, batch by batch, into the running sums and consume
// them (reset the folded entries): d = q * 1e-9 / (mass * n), s1 += d, s2 += d^2
// (kernels.py:804-852).  A lane owns half a dirty sector (two entries, 16-byte
// loads) and goes through those of the wave's maps whose own bitmap has the sector,
// in batch order (most sectors are hit in one or two of the batches), the next
// map's quanta on their way while the current ones are added in registers; the
// sums cross memory once per wave.  kFinal: the wave holds every batch of the run,
// so every touched sector is dirty here and the mean, sigma and column maximum are
// written at once (finalize_sparse_kernel otherwise).  What bounds it: the latency
// of scattered 32-byte sectors, some 1e7 of them per wave of the 100-column 128^3
// Dij, then the issue of the float64 arithmetic (one reciprocal per entry instead
// of a division per entry and batch).
// kDivide: masses that no tissue has (infinite, say) are divided by as they are; in
// one kernel with the reciprocal the division's registers spill (2.17 -> 2.35 ms).
constexpr int kWaveMaps = 32;  // the most maps of a wave

template <bool kFinal, bool kDivide>
__global__ void __launch_bounds__(kReduceThreads, 4)
fold_sparse_kernel(unsigned long long* __restrict__ edep, const double* __restrict__ mass,
                   const double* __restrict__ col_nhist, FoldShape f, double* __restrict__ s1,
                   double* __restrict__ s2, unsigned int* __restrict__ dirty,
                   unsigned int* __restrict__ touched, int n_batches,
                   unsigned long long* __restrict__ col_max_bits, unsigned long long* __restrict__ total_q) {
    __shared__ unsigned int map_word[kReduceThreads / 32][kWaveMaps][32];  // the part's words, map by map
    const int lane = threadIdx.x & 31;
    unsigned int (*mine)[32] = map_word[threadIdx.x >> 5];
    const long long map_words = f.map_entries / kWordEntries;
    const double n = (double)n_batches;
    // a part's words lie at part * words (the columns' words follow one another)
    auto dirty_word = [&](unsigned int part, unsigned int end) {
        unsigned int w = 0u;
        if (part < end && lane < f.words) {
            const unsigned int* p = dirty + (long long)part * f.words + lane;
#pragma unroll 4
            for (int m = 0; m < f.n_maps; ++m) w |= p[m * map_words];
        }
        return w;
    };
    unsigned long long local = 0;
    for (unsigned int t = claim_parts(f), end; t < f.n_parts; t = claim_parts(f))
    for (unsigned int w_next = dirty_word(t, end = min(t + f.claim, f.n_parts)); t < end; ++t) {
        const unsigned int w = w_next;
        w_next = dirty_word(t + 1u, end);
        if (__ballot_sync(0xffffffffu, w != 0u) == 0u) continue;
        const long long widx = (long long)t * f.words + lane;
        const long long col = t / f.parts_per_col;
        const long long word0 = (t - col * f.parts_per_col) * f.words;  // in the column
        const unsigned int tw = lane < f.words ? touched[widx] : 0u;
#pragma unroll 4
        for (int m = 0; m < f.n_maps; ++m) mine[m][lane] = lane < f.words ? dirty[m * map_words + widx] : 0u;
        __syncwarp();
        const int incl = warp_inclusive_scan(__popc(w));
        const int total = __shfl_sync(0xffffffffu, incl, 31);
        const double nh = col_nhist[col];
        unsigned long long best = 0;
        for (int k0 = 0; k0 < total; k0 += 16) {
            const int k = k0 + (lane >> 1);
            int bit;
            const int j = nth_set_sector(w, incl, k, bit);
            const unsigned int twj = __shfl_sync(0xffffffffu, tw, j);
            if (k >= total) continue;
            const long long v = (word0 + j) * kWordEntries + bit * kSectorEntries + 2 * (lane & 1);
            const long long at = col * f.stride + v;
            unsigned int maps = 0u;  // the maps that hold this sector
#pragma unroll 4
            for (int m = 0; m < f.n_maps; ++m) maps |= ((mine[m][j] >> bit) & 1u) << m;
            auto quanta = [&](unsigned int left) {
                return reinterpret_cast<ulonglong2*>(edep + (__ffs((int)left) - 1) * f.map_entries + at);
            };
            ulonglong2* q_at = quanta(maps);
            ulonglong2 q = *q_at;
            double2 a = make_double2(0.0, 0.0), b = a, y = a;
            if ((twj >> bit) & 1u) {  // folded before
                a = *reinterpret_cast<const double2*>(s1 + at);
                b = *reinterpret_cast<const double2*>(s2 + at);
            }
            if (v < f.n_vox) y.x = mass[v];
            if (v + 1 < f.n_vox) y.y = mass[v + 1];
            const bool some_x = y.x > 0.0, some_y = y.y > 0.0;  // no mass: no dose
            y.x = some_x ? __dmul_rn(y.x, nh) : 0.0;
            y.y = some_y ? __dmul_rn(y.y, nh) : 0.0;
            const double rx = !kDivide && y.x > 0.0 ? __drcp_rn(y.x) : 0.0;
            const double ry = !kDivide && y.y > 0.0 ? __drcp_rn(y.y) : 0.0;
            auto dose = [](unsigned long long quanta, bool some, double by, double r) {
                const double energy = __dmul_rn((double)(long long)quanta, kQuantum);
                if constexpr (kDivide) return some && quanta != 0ull ? __ddiv_rn(energy, by) : 0.0;
                else return divide_by(energy, by, r);
            };
            for (;;) {
                maps &= maps - 1u;
                ulonglong2* const next_at = maps ? quanta(maps) : q_at;
                ulonglong2 q_next = q;
                if (maps) q_next = *next_at;
                if ((q.x | q.y) != 0ull) *q_at = make_ulonglong2(0ull, 0ull);
                const double dx = dose(q.x, some_x, y.x, rx);
                const double dy = dose(q.y, some_y, y.y, ry);
                a.x = __dadd_rn(a.x, dx);
                a.y = __dadd_rn(a.y, dy);
                b.x = __dadd_rn(b.x, __dmul_rn(dx, dx));
                b.y = __dadd_rn(b.y, __dmul_rn(dy, dy));
                local += q.x + q.y;
                if (maps == 0u) break;
                q = q_next;
                q_at = next_at;
            }
            if constexpr (kFinal) {
                finalize_entry(a.x, b.x, n, n_batches);
                finalize_entry(a.y, b.y, n, n_batches);
                const unsigned long long bx = (unsigned long long)__double_as_longlong(a.x);
                const unsigned long long by = (unsigned long long)__double_as_longlong(a.y);
                best = max(best, max(bx, by));  // as column_max
            }
            *reinterpret_cast<double2*>(s1 + at) = a;
            *reinterpret_cast<double2*>(s2 + at) = b;
        }
        if (w != 0u) {
            for (int m = 0; m < f.n_maps; ++m)
                if (mine[m][lane]) dirty[m * map_words + widx] = 0u;
            touched[widx] = tw | w;
        }
        __syncwarp();
        if constexpr (kFinal) column_max(best, col_max_bits + col);
    }
    local = warp_sum_u64(local);
    if (lane == 0 && local) atomicAdd(total_q, local);
}

// Mean and sigma of the touched sectors, in place, with the column maximum of
// the mean (one atomic per warp and part).
__global__ void __launch_bounds__(kReduceThreads, 3)
finalize_sparse_kernel(double* __restrict__ s1, double* __restrict__ s2, FoldShape f, int n_batches,
                       const unsigned int* __restrict__ touched,
                       unsigned long long* __restrict__ col_max_bits) {
    const int lane = threadIdx.x & 31;
    const double n = (double)n_batches;
    auto word = [&](unsigned int part, unsigned int end) {
        return part < end && lane < f.words ? touched[(long long)part * f.words + lane] : 0u;
    };
    for (unsigned int t = claim_parts(f), end; t < f.n_parts; t = claim_parts(f))
    for (unsigned int w_next = word(t, end = min(t + f.claim, f.n_parts)); t < end; ++t) {
        const unsigned int w = w_next;
        w_next = word(t + 1u, end);
        if (__ballot_sync(0xffffffffu, w != 0u) == 0u) continue;
        const long long col = t / f.parts_per_col;
        const long long word0 = (t - col * f.parts_per_col) * f.words;
        const int incl = warp_inclusive_scan(__popc(w));
        const int total = __shfl_sync(0xffffffffu, incl, 31);
        unsigned long long best = 0ull;
        // the next sector's sums are on their way while this one's are finalized
        auto sector = [&](int k) {
            int bit;
            const int j = nth_set_sector(w, incl, k, bit);
            return k < total ? col * f.stride + (word0 + j) * kWordEntries + bit * kSectorEntries : -1ll;
        };
        SectorD a, b;
        long long at = sector(lane);
        if (at >= 0) {
            a.load(s1 + at);
            b.load(s2 + at);
        }
        for (int k0 = 0; k0 < total; k0 += 32) {
            SectorD a_next, b_next;
            const long long at_next = sector(k0 + 32 + lane);
            if (at_next >= 0) {
                a_next.load(s1 + at_next);
                b_next.load(s2 + at_next);
            }
            if (at >= 0) {
#pragma unroll
                for (int e = 0; e < kSectorEntries; ++e) {
                    finalize_entry(a.v[e], b.v[e], n, n_batches);
                    const unsigned long long bits = (unsigned long long)__double_as_longlong(a.v[e]);
                    best = bits > best ? bits : best;
                }
                a.store(s1 + at);
                b.store(s2 + at);
            }
            at = at_next;
            a = a_next;
            b = b_next;
        }
        column_max(best, col_max_bits + col);
    }
}

// Kept entries of the touched sectors of one (column, tile); one warp each.
__global__ void __launch_bounds__(kReduceThreads)
count_kept_sparse_kernel(const double* __restrict__ mean, long long n_vox, long long stride,
                         int tiles_per_col, long long n_tiles, double truncation,
                         const unsigned long long* __restrict__ col_max_bits,
                         const unsigned int* __restrict__ touched,
                         unsigned int* __restrict__ tile_counts) {
    const int lane = threadIdx.x & 31;
    const long long t = (long long)blockIdx.x * (kReduceThreads / 32) + (threadIdx.x >> 5);
    if (t >= n_tiles) return;
    const unsigned int w = touched[t * 32 + lane];
    unsigned int c = 0;
    if (__ballot_sync(0xffffffffu, w != 0u) != 0u) {
        const int incl = warp_inclusive_scan(__popc(w));
        const int total = __shfl_sync(0xffffffffu, incl, 31);
        const long long col = t / tiles_per_col;
        const long long tile_v0 = (t - col * tiles_per_col) * (long long)kTileVoxels;
        const double thr = __dmul_rn(truncation, __longlong_as_double((long long)col_max_bits[col]));
        const double* a = mean + col * stride;
        for (int k0 = 0; k0 < total; k0 += 32) {
            const int k = k0 + lane;
            int bit;
            const int j = nth_set_sector(w, incl, k, bit);
            if (k >= total) continue;
            const long long v0 = tile_v0 + (long long)j * kWordEntries + bit * kSectorEntries;
#pragma unroll
            for (int e = 0; e < kSectorEntries; ++e) {
                const long long v = v0 + e;
                if (v < n_vox) c += keep_entry(a[v], thr);
            }
        }
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) c += __shfl_xor_sync(0xffffffffu, c, off);
    if (lane == 0) tile_counts[t] = c;
}

// Write the kept entries of one (column, tile) at the tile's CSC offset, in
// ascending voxel order (sector order, then entry order): the order
// np.flatnonzero gives on the host.  One warp each.
__global__ void __launch_bounds__(kReduceThreads)
compact_sparse_kernel(const double* __restrict__ mean, const double* __restrict__ sigma,
                      long long n_vox, long long stride, int tiles_per_col, long long n_tiles,
                      double truncation, const unsigned long long* __restrict__ col_max_bits,
                      const unsigned int* __restrict__ touched,
                      const unsigned long long* __restrict__ tile_offsets,
                      long long* __restrict__ out_idx, double* __restrict__ out_dose,
                      double* __restrict__ out_sigma) {
    const int lane = threadIdx.x & 31;
    const long long t = (long long)blockIdx.x * (kReduceThreads / 32) + (threadIdx.x >> 5);
    if (t >= n_tiles) return;
    const unsigned int w = touched[t * 32 + lane];
    if (__ballot_sync(0xffffffffu, w != 0u) == 0u) return;
    const int incl = warp_inclusive_scan(__popc(w));
    const int total = __shfl_sync(0xffffffffu, incl, 31);
    const long long col = t / tiles_per_col;
    const long long tile_v0 = (t - col * tiles_per_col) * (long long)kTileVoxels;
    const double thr = __dmul_rn(truncation, __longlong_as_double((long long)col_max_bits[col]));
    const double* a = mean + col * stride;
    const double* b = sigma + col * stride;
    unsigned long long cursor = tile_offsets[t];
    for (int k0 = 0; k0 < total; k0 += 32) {
        const int k = k0 + lane;
        int bit;
        const int j = nth_set_sector(w, incl, k, bit);
        const long long v0 = tile_v0 + (long long)j * kWordEntries + bit * kSectorEntries;
        double m[kSectorEntries];
        unsigned int keep = 0u;
#pragma unroll
        for (int e = 0; e < kSectorEntries; ++e) {
            const long long v = v0 + e;
            m[e] = (k < total && v < n_vox) ? a[v] : 0.0;
            if (k < total && v < n_vox && keep_entry(m[e], thr)) keep |= 1u << e;
        }
        const int n_keep = __popc(keep);
        const int end = warp_inclusive_scan(n_keep);
        unsigned long long pos = cursor + (unsigned long long)(end - n_keep);
#pragma unroll
        for (int e = 0; e < kSectorEntries; ++e) {
            if (keep & (1u << e)) {
                out_idx[pos] = v0 + e;
                out_dose[pos] = m[e];
                out_sigma[pos] = b[v0 + e];
                ++pos;
            }
        }
        cursor += (unsigned long long)__shfl_sync(0xffffffffu, end, 31);
    }
}

// Set every word of a bitmap (the dense entry points mark every sector).
__global__ void fill_u32_kernel(unsigned int* p, long long n, unsigned int v) {
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) p[i] = v;
}

// One entry of each of kTileStep * 32 consecutive ones per lane and step, loaded
// together (columns need not be 16-byte aligned: their length may be odd).
constexpr int kTileStep = 8;

// Column maxima of an already finalized mean map with columns `stride` entries
// apart, and (tile_max not null) the maximum of every tile, as the bits of a
// non-negative double.  One warp per (tile, column) (grid: x = tiles / 8, y = column);
// bound by the one read of the map: 16 loads of 8 bytes in flight per lane.
__global__ void __launch_bounds__(kReduceThreads)
colmax_kernel(const double* __restrict__ mean, long long n_vox, long long stride, int n_tiles,
              unsigned long long* __restrict__ col_max_bits, unsigned long long* __restrict__ tile_max) {
    const long long col = blockIdx.y;
    const int tile = blockIdx.x * (kReduceThreads / 32) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (tile >= n_tiles) return;  // warp-uniform
    const long long start = (long long)tile * kTileVoxels;
    const double* a = mean + col * stride + start;
    const int count = (int)min((long long)kTileVoxels, n_vox - start);
    double top = 0.0;  // only positive entries count
    if (count == kTileVoxels) {
        for (int v0 = lane; v0 < kTileVoxels; v0 += 2 * kTileStep * 32) {
            double m[2 * kTileStep];
#pragma unroll
            for (int i = 0; i < 2 * kTileStep; ++i) m[i] = __ldcs(a + v0 + 32 * i);
#pragma unroll
            for (int i = 0; i < 2 * kTileStep; ++i) top = m[i] > top ? m[i] : top;
        }
    } else {
        for (int v = lane; v < count; v += 32) top = a[v] > top ? a[v] : top;
    }
    unsigned long long best = (unsigned long long)__double_as_longlong(top);
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) best = max(best, __shfl_xor_sync(0xffffffffu, best, off));
    if (lane == 0) {
        if (best) atomicMax(col_max_bits + col, best);
        if (tile_max) tile_max[col * n_tiles + tile] = best;
    }
}

// Count the kept entries of one (column, tile); one warp each.  A tile whose
// maximum is below the threshold is not read (most of a beamlet's column).
__global__ void __launch_bounds__(kReduceThreads)
count_kept_kernel(const double* __restrict__ mean, long long n_vox, int n_tiles, double truncation,
                  const unsigned long long* __restrict__ col_max_bits,
                  const unsigned long long* __restrict__ tile_max, unsigned int* __restrict__ tile_counts) {
    const long long col = blockIdx.y;
    const int tile = blockIdx.x * (kReduceThreads / 32) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (tile >= n_tiles) return;
    const long long start = (long long)tile * kTileVoxels;
    const double thr = __dmul_rn(truncation, __longlong_as_double((long long)col_max_bits[col]));
    unsigned int c = 0;
    if (keep_entry(__longlong_as_double((long long)tile_max[col * n_tiles + tile]), thr)) {
        const double* a = mean + col * n_vox + start;
        const int count = (int)min((long long)kTileVoxels, n_vox - start);
        for (int v0 = 0; v0 < count; v0 += kTileStep * 32) {
            double m[kTileStep];
#pragma unroll
            for (int i = 0; i < kTileStep; ++i) {
                const int v = v0 + 32 * i + lane;
                m[i] = v < count ? a[v] : 0.0;
            }
#pragma unroll
            for (int i = 0; i < kTileStep; ++i) c += keep_entry(m[i], thr);
        }
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) c += __shfl_xor_sync(0xffffffffu, c, off);
    if (lane == 0) tile_counts[col * n_tiles + tile] = c;
}

// Write the kept entries of one (column, tile) in ascending voxel order at the
// tile's offset: the same order np.flatnonzero gives on the host.  One warp each;
// tiles without one are not read.
__global__ void __launch_bounds__(kReduceThreads)
compact_kernel(const double* __restrict__ mean, const double* __restrict__ sigma, long long n_vox,
               int n_tiles, double truncation, const unsigned long long* __restrict__ col_max_bits,
               const unsigned int* __restrict__ tile_counts,
               const unsigned long long* __restrict__ tile_offsets, long long* __restrict__ out_idx,
               double* __restrict__ out_dose, double* __restrict__ out_sigma) {
    const long long col = blockIdx.y;
    const int tile = blockIdx.x * (kReduceThreads / 32) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (tile >= n_tiles) return;
    if (tile_counts[col * n_tiles + tile] == 0u) return;
    const long long start = (long long)tile * kTileVoxels;
    const double thr = __dmul_rn(truncation, __longlong_as_double((long long)col_max_bits[col]));
    const double* a = mean + col * n_vox + start;
    const double* b = sigma + col * n_vox + start;
    const int count = (int)min((long long)kTileVoxels, n_vox - start);
    unsigned long long cursor = tile_offsets[col * n_tiles + tile];
    for (int v0 = 0; v0 < count; v0 += kTileStep * 32) {
        double m[kTileStep];
#pragma unroll
        for (int i = 0; i < kTileStep; ++i) {
            const int v = v0 + 32 * i + lane;
            m[i] = v < count ? a[v] : 0.0;
        }
#pragma unroll
        for (int i = 0; i < kTileStep; ++i) {
            const bool k = keep_entry(m[i], thr);
            const unsigned int ballot = __ballot_sync(0xffffffffu, k);
            if (k) {
                const int v = v0 + 32 * i + lane;
                const unsigned long long pos = cursor + __popc(ballot & ((1u << lane) - 1u));
                out_idx[pos] = start + v;
                out_dose[pos] = m[i];
                out_sigma[pos] = b[v];
            }
            cursor += __popc(ballot);
        }
    }
}

}  // namespace pmc
