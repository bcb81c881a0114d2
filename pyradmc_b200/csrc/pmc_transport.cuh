// pmc_transport.cuh — the persistent photon and electron transport kernels.
//
// Behavioural spec: photon_kernel / electron_kernel of
// pyradmc/backends/warp/kernels.py:1171-1885, which mirror the reference loops
// transport/photon.py:100-282 and transport/electron.py:207-482 statement for
// statement.  The structure is B200-first rather than a translation:
//   * persistent grids (a multiple of the SM count) with per-lane refill: a
//     lane whose particle ends takes the next one of the input queue at once, so
//     no lane idles behind the longest particle of its warp;
//   * primaries are generated at full warp width and queued (generate_kernel);
//   * queue rotation, the primary admission window and the "work left" flag
//     are advanced on the device by the last block of each kernel, so a whole
//     wave of batches drains without one host round trip (and inside one CUDA graph);
//   * no counter that other blocks use is touched per particle: input is claimed
//     32 particles at a time and output slots are taken in chunks;
//   * energy books and event counters accumulate in shared memory and reach
//     global memory once per block.
#pragma once

#include <cooperative_groups.h>

#include <type_traits>

#include "pmc_common.cuh"
#include "pmc_physics.cuh"
#include "pmc_reduce.cuh"
#include "pmc_stack.cuh"

namespace pmc {

namespace cg = cooperative_groups;

// Flags raised on the device and reported by the host after a batch.
constexpr int kFlagOverflow = 1;
constexpr int kFlagStepCap = 2;
constexpr int kFlagRoundCap = 4;

// A counter on a cache line of its own: atomics on one line pass one at a time.
struct alignas(128) Counter32 {
    unsigned int v;
};

// Device-resident scheduling state of one drain (a wave of statistical batches).
// A queue (P0, P1, E0, E1) fills from both ends: whole chunks and the window of
// fresh primaries from slot 0 up (bottom), single particles from its last slot
// down (top).  Some bottom slots stay dead (marked; counted in `dead`).
struct Sched {
    Counter32 bottom[4];
    Counter32 top[4];
    Counter32 head[4];              // fetch heads
    Counter32 dead[4];
    int p_in, e_in;                 // input photon / electron queue (0/1)
    unsigned int window_base;       // first slot of the round's fresh primaries
    unsigned long long cursor;      // next primary of the wave
    unsigned long long limit;       // admission limit of the current round
    unsigned long long block_end;   // primaries in the wave
    unsigned long long budget;      // primaries admitted per round
    unsigned int blocks_done;
    int flags;
    int remaining;                  // 1 while work is left
    int batch;                      // first batch of the wave
    long long rounds;               // rounds of the current wave
    long long total_rounds;         // rounds of the whole call (not reset per wave)
    long long max_rounds;
    unsigned long long cond_handle; // CUDA graph conditional handle (0: host loop)
};

// One beamlet (or one mixture component of a beamlet) of the record
// generator, 64 bytes:
//   lattice: a = (x_lo, x_extent, y_lo, y_extent), b = (z0, energy, -, -)
//   fan:     a = (focal, width_u), b = (aperture centre, width_v),
//            c = (u axis, first spectrum entry), d = (v axis, -)
// d.w holds the kind (0 lattice, 1 fan) in bit 0 and the fan's spectrum bin
// count above it, as integer bits.  Spectra are concatenated in segments of
// n_bins + 1 entries that start at the same index in the edge and the
// cumulative arrays (the cumulative segment's last entry is unused).
struct __align__(16) BeamletRec {
    float4 a, b, c, d;
};

// Primary generator of the current group (device-resident).
struct GenDesc {
    int type;           // 0 pencil, 1 parallel/lattice, 2 spectral fan, 3 upload, 4 records,
                        // 5 resident phase space
    int kind;           // particle kind of analytic primaries
    int forward;        // 1: open-field run (history = batch * per_batch + t)
    int correlated;
    int group;          // columns in this group
    int n_bins;
    float energy;
    float px, py, pz, dx, dy, dz;       // pencil
    float z0;                            // parallel / lattice
    float fx, fy, fz;                    // spectral focal point
    float uax, uay, uaz, vax, vay, vaz;  // aperture axes
    float width_u, width_v;
    long long per_batch_fwd;             // forward: histories per batch
    unsigned long long wave_block;       // primaries of one batch when a wave holds several, else 0
    const long long* pb_prefix;          // [group+1] exclusive prefix of per-batch counts
    const long long* per_batch;          // [group]
    const long long* hist_offset;        // [group] first global history of each beamlet
    const float* x_lo;                   // [group] lattice bounds
    const float* x_ext;
    const float* y_lo;
    const float* y_ext;
    const float* cx;                     // [group] spectral centres
    const float* cy;
    const float* cz;
    const float* edges;                  // [n_bins+1]
    const float* cdf;                    // [n_bins]
    const int* up_kind;                  // upload route, [n_histories]
    const float* up_energy;
    const float* up_pos;
    const float* up_dir;
    const float* up_weight;
    int book_emitted;                    // spectral/upload: book emitted energy per primary
    long long n_records;                 // resident phase space: records in up_*
    const BeamletRec* recs;              // records: [group][n_comp]
    const float* comp_cdf;               // records: [n_comp] mixture selection
    int n_comp;
    int masked;                          // spectral fan through a transmission mask
    int mask_n_u, mask_n_v;
    const float* mask;                   // [mask_n_u * mask_n_v]
    float mcx, mcy, mcz;                 // mask plane centre
    float mux, muy, muz, mvx, mvy, mvz;  // mask pixel axes
    float mask_wu, mask_wv;
    int stacked;                         // collimated: weight by the stack transmission
    pmc_head::Stack stack;
    pmc_head::Mu stack_mu;               // macroscopic attenuation, one row per device
};

struct Counters {
    unsigned long long flights, interactions, substeps, deposits, pushes, primaries;
    long long escaped, unscored, deposited, emitted, violations;
};

// Cylindrical scoring bins (geometry/cylinder.py): depth along z by radial
// shell about an axis parallel to z, edges in float32 as the Warp kernels hold
// them, radial edges squared.
struct CylInfo {
    float ax, ay;             // axis
    float z_lo, z_hi;         // first and last depth edge
    float r_in_sq, r_out_sq;  // first and last squared radial edge
    int n_depth, n_shells;
    const float* z_edges;     // [n_depth + 1]
    const float* r_edges_sq;  // [n_shells + 1]
};

struct TransportParams {
    GridInfo gi;          // transport grid
    GridInfo si;          // scoring grid (score_mode 0)
    int score_mode;       // 0 rectilinear, 1 cylindrical
    CylInfo cyl;          // scoring bins (score_mode 1)
    const float2* vox;    // (density, material bits) per transport voxel
    Tables tab;
    Slot* q[4];           // P0, P1, E0, E1
    unsigned int capacity;     // particles a queue may hold
    unsigned int slots;        // slots behind it: capacity and room for dead ones
    int window_el;             // fresh primaries enter the electron queue (a charged source)
    Sched* sched;
    const GenDesc* gen;
    unsigned long long* edep;  // [batch of the wave][group][col_stride] int64 quanta
    unsigned int* dirty;       // sector bitmap of edep (pmc_reduce.cuh)
    long long col_stride;      // entries per column: scoring voxels rounded up to a tile
    Counters* counters;
    uint32_t seed_lo, seed_hi;
    PhiloxKeys keys;      // of the seed
    float pcut, ecut;
    float step_fraction;
    float deposit_resolution;
    int transport_electrons;
    int msc_gs;
    int dose_to_water;
    int split_n;
    int max_steps;
    int tail_steps;       // steps a lane may still take once its round's input ran dry
};

// ---- per-block books ------------------------------------------------------------
struct BlockBooks {
    unsigned long long flights, interactions, substeps, deposits, pushes, primaries;
    long long escaped, unscored, deposited, emitted, violations;
    unsigned long long dead;  // slots a generator block left dead
};

__device__ __forceinline__ long long quantize_signed(float amount) {
    return (long long)floor((double)amount * kInvQuantum + 0.5);
}

__device__ __forceinline__ void book_add(long long* slot, long long v) {
    if (v != 0) atomicAdd((unsigned long long*)slot, (unsigned long long)v);
}

// kernels.py:459 _spr_factor: restricted-stopping ratio water/medium, exactly 1
// under dose-to-medium and for water deposits.
__device__ __forceinline__ float spr_factor(const TransportParams& P, float e, int mat) {
    if (P.dose_to_water == 0 || mat == kWater) return 1.0f;
    const LogIdx li = log_index(fmaxf(e, P.ecut), P.tab.e_log_min, P.tab.e_inv_dlog, P.tab.n_points);
    const float sw = lerp1(P.tab.ec + (long long)kWater * P.tab.n_points, li);
    const float sm = lerp1(P.tab.ec + (long long)mat * P.tab.n_points, li);
    return sw / sm;
}

// Where a deposit's quanta go.  DirectSink issues one atomic per deposit;
// HeldSink keeps one pending (entry, quanta) pair in registers and merges the
// next deposit into it when it lands in the same entry — an electron's two
// half-substep deposits and its next substep's usually do — so a run of
// deposits into one voxel costs one atomic.  Integer sums: merging is exact.
// Every atomic also marks its entry's sector in the dirty bitmap, the only
// sectors the batch fold visits.  Entries are named by their bin in the
// particle's column; the column's offset is recomputed at each atomic instead of
// being held in two registers for the particle's whole life.
struct DirectSink {
    unsigned int n = 0;  // atomics issued
    template <typename Bin>
    __device__ __forceinline__ void add(const TransportParams& P, int beamlet, Bin bin, unsigned long long q) {
        const long long flat = (long long)beamlet * P.col_stride + bin;
        atomicAdd(P.edep + flat, q);
        mark_dirty(P.dirty, flat);
        ++n;
    }
};

template <typename Bin>
struct HeldSink {
    Bin bin = -1;
    unsigned long long q = 0;
    unsigned int n = 0;
    __device__ __forceinline__ void add(const TransportParams& P, int beamlet, Bin at, unsigned long long quanta) {
        if (at == bin) {
            q += quanta;
            return;
        }
        release(P, beamlet);
        bin = at;
        q = quanta;
    }
    // The pending deposit reaches the map: before the lane changes its beamlet.
    __device__ __forceinline__ void release(const TransportParams& P, int beamlet) {
        if (q != 0ull) {
            const long long flat = (long long)beamlet * P.col_stride + bin;
            atomicAdd(P.edep + flat, q);
            mark_dirty(P.dirty, flat);
            ++n;
        }
        bin = -1;
        q = 0ull;
    }
};

// edge_bin_index (geometry/cylinder.py): the bin k with edges[k] <= v <
// edges[k + 1], clamped into [0, n - 1]; the caller has checked containment.
__device__ __forceinline__ int edge_bin_index(float v, const float* edges, int n) {
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (v >= __ldg(edges + mid)) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// kernels.py:492 _scoring_index: the flat scoring bin of a position, or -1
// when the scoring geometry excludes it (half-open on every axis and shell).
__device__ __forceinline__ long long scoring_index(const TransportParams& P, float x, float y,
                                                   float z) {
    if (P.score_mode == 0) return point_inside(x, y, z, P.si) ? flat_index(x, y, z, P.si) : -1;
    const CylInfo& c = P.cyl;
    if (z < c.z_lo || z >= c.z_hi) return -1;
    const float dx = x - c.ax, dy = y - c.ay;
    const float r2 = dx * dx + dy * dy;
    if (r2 < c.r_in_sq || r2 >= c.r_out_sq) return -1;
    const int depth = edge_bin_index(z, c.z_edges, c.n_depth);
    const int shell = edge_bin_index(r2, c.r_edges_sq, c.n_shells);
    return (long long)depth * c.n_shells + shell;
}

// Bins of a column: 32-bit in the kPlain kernels (fewer than 2^31 voxels).
template <bool kPlain>
using BinOf = std::conditional_t<kPlain, int, long long>;

__device__ __forceinline__ long long quantize(float amount) {
    return (long long)((double)amount * kInvQuantum + 0.5);
}

// kernels.py:536 _deposit: quantize once, route by position into the scoring
// grid of this particle's column, or into the unscored book.  kPlain: the caller
// has the position's bin already, and the factor is exactly 1.
template <bool kPlain, class Sink>
__device__ __forceinline__ void deposit(const TransportParams& P, BlockBooks& B, int beamlet, float x,
                                       float y, float z, int voxel, float amount, float factor, Sink& sink) {
    if constexpr (kPlain) {
        const long long q = quantize(amount);
        if (q != 0) sink.add(P, beamlet, voxel, (unsigned long long)q);
    } else {
        const long long idx = scoring_index(P, x, y, z);
        if (idx >= 0) {
            const long long q =
                (long long)((double)amount * (double)factor * kInvQuantum + 0.5);
            if (q != 0) sink.add(P, beamlet, idx, (unsigned long long)q);
            if (P.dose_to_water) book_add(&B.deposited, quantize(amount));
        } else {
            book_add(&B.unscored, quantize(amount));
        }
    }
}

__device__ __forceinline__ void escape(BlockBooks& B, float amount) {
    book_add(&B.escaped, quantize_signed(amount));
}

// flat_index of a grid of fewer than 2^31 voxels.
__device__ __forceinline__ int flat_index32(float x, float y, float z, const GridInfo& g) {
    const int ix = axis_index(x, g.x_lo, g.sx, g.nx);
    const int iy = axis_index(y, g.y_lo, g.sy, g.ny);
    const int iz = axis_index(z, g.z_lo, g.sz, g.nz);
    return (ix * g.ny + iy) * g.nz + iz;
}
template <bool kPlain>
__device__ __forceinline__ BinOf<kPlain> voxel_of(float x, float y, float z, const GridInfo& g) {
    if constexpr (kPlain) return flat_index32(x, y, z, g);
    else return flat_index(x, y, z, g);
}

// kernels.py:600 _deposit_or_escape: escape is decided on the transport grid.
template <bool kPlain, class Sink>
__device__ __forceinline__ void deposit_or_escape(const TransportParams& P, BlockBooks& B, int beamlet,
                                                  float x, float y, float z, float amount, float factor,
                                                  Sink& sink) {
    if (amount <= 0.0f) return;
    if (point_inside(x, y, z, P.gi))
        deposit<kPlain>(P, B, beamlet, x, y, z, kPlain ? flat_index32(x, y, z, P.gi) : 0, amount, factor, sink);
    else escape(B, amount);
}

// kernels.py:631 _deposit_spread: equal pieces at piece midpoints (kPlain: one).
template <bool kPlain, class Sink>
__device__ __forceinline__ void deposit_spread(const TransportParams& P, BlockBooks& B, int beamlet, float x,
                                               float y, float z, float ux, float uy, float uz, float length,
                                               float amount, float factor, Sink& sink) {
    const int n = kPlain ? 1 : substep_pieces(length, P.deposit_resolution);
    const float share = kPlain ? amount : amount / (float)n;
    const float piece = kPlain ? length : length / (float)n;
    for (int k = 0; k < n; ++k) {
        const float t = ((float)k + 0.5f) * piece;
        deposit_or_escape<kPlain>(P, B, beamlet, x + ux * t, y + uy * t, z + uz * t, share, factor, sink);
    }
}

// ---- queue slots ------------------------------------------------------------------
// One atomic on a queue's counter per pushing group of lanes, and one per refill,
// held the transport kernels to about one such atomic per nanosecond over the
// whole GPU (two thirds of the photon kernel's stalls on a 1.2e6-primary round).
// So a block takes slots kChunk at a time: its word (shared memory) is the chunk's
// number above kOffBits bits of fill.  A group adds its size; the group that takes
// a chunk's last slot opens the next one and publishes it, and groups that come
// while it does so go to the top of the queue instead of waiting.  At most one add
// per lane can follow the chunk's end before the next chunk is published, so the
// fill never carries into the chunk number.  The slots a block leaves unused are
// marked dead.
constexpr unsigned int kChunk = 128;
constexpr int kOffBits = 11;
constexpr unsigned int kOffMask = (1u << kOffBits) - 1u;
constexpr unsigned int kChunkedSlots = kChunk << (32 - kOffBits);  // slots a chunk number can name
constexpr uint32_t kDeadMeta = 0xffffffffu;
static_assert(kChunk + 1024 < kOffMask, "a block's lanes fit above the chunk in the fill field");

__device__ __forceinline__ unsigned int round_to_chunk(unsigned long long n) {
    return (unsigned int)((n + kChunk - 1) / kChunk * kChunk);
}

// One round of a kernel as its blocks see it, in shared memory: the particles of
// its input queue, and the two queues it pushes to with the block's chunk of each
// (chunk number above kOffBits bits of fill; kChunk and more: closed, slots are
// taken singly from the top).
struct Round {
    int q_in, q_out[2];
    unsigned int n_bottom, n;  // particles from the bottom of the input queue, in all
    unsigned int claim;        // particles a warp claims at a time
    uint32_t chunk[2];
    unsigned int pushes;
};

// One thread of the block.  Chunks (of the queues in `chunk_mask`) pay where a
// round is long and the slots left unused do not count, at 512 input particles
// per block and more; small rounds take single slots, and claim few particles at
// a time, so that every warp gets some.
__device__ __forceinline__ void open_round(const TransportParams& P, Round& R, int q_in, int q_out0, int q_out1,
                                           unsigned int chunk_mask) {
    Sched* S = P.sched;
    R.q_in = q_in;
    R.q_out[0] = q_out0;
    R.q_out[1] = q_out1;
    const unsigned int b = S->bottom[q_in].v, t = S->top[q_in].v;
    R.n_bottom = min(b, P.slots);
    R.n = R.n_bottom + min(t, P.slots - R.n_bottom);
    if ((unsigned long long)b + t > (unsigned long long)P.capacity + S->dead[q_in].v) {  // too many live ones
        atomicOr(&S->flags, kFlagOverflow);
        R.n = R.n_bottom = 0u;
    }
    const unsigned int warps = gridDim.x * (blockDim.x / 32u);
    R.claim = R.n / warps >= 128u ? 32u : R.n / warps >= 16u ? 4u : 1u;
    const bool chunked = R.n >= 512u * gridDim.x && P.slots <= kChunkedSlots;
    for (int k = 0; k < 2; ++k)
        R.chunk[k] = chunked && (chunk_mask >> k & 1u)
                         ? atomicAdd(&S->bottom[R.q_out[k]].v, kChunk) / kChunk << kOffBits
                         : kChunk;
    R.pushes = 0u;
}

// A single slot of queue qi for every lane that gets here together, from the top
// down; P.slots when there is none.
__device__ __forceinline__ unsigned int single_slot(const TransportParams& P, int qi) {
    cg::coalesced_group g = cg::coalesced_threads();
    unsigned int base = 0u;
    if (g.thread_rank() == 0) base = atomicAdd(&P.sched->top[qi].v, (unsigned int)g.size());
    base = g.shfl(base, 0) + (unsigned int)g.thread_rank();
    return base < P.slots ? P.slots - 1u - base : P.slots;
}

// A slot of output queue k for every lane that gets here together; P.slots and up
// when there is none.
__device__ __forceinline__ unsigned int claim_slot(const TransportParams& P, Round& R, int k) {
    cg::coalesced_group g = cg::coalesced_threads();
    const unsigned int n = (unsigned int)g.size(), r = (unsigned int)g.thread_rank();
    unsigned int first = 0u, rest = 0u, served = 0u;  // served lanes from `first`, the others from `rest`
    if (r == 0u) {
        uint32_t* word = &R.chunk[k];
        bool single = true;
        if ((*(volatile uint32_t*)word & kOffMask) < kChunk) {
            const uint32_t w = atomicAdd(word, n);
            const unsigned int off = w & kOffMask;
            if (off < kChunk) {
                first = (w >> kOffBits) * kChunk + off;
                served = min(n, kChunk - off);
                single = false;
                if (off + n >= kChunk) {  // the chunk's last slot: open the next
                    rest = atomicAdd(&P.sched->bottom[R.q_out[k]].v, kChunk);
                    atomicExch(word, (rest / kChunk << kOffBits) | (n - served));
                }
            }
        }
        if (single) {
            rest = atomicAdd(&P.sched->top[R.q_out[k]].v, n);
            served = 0x100u;
        }
        atomicAdd(&R.pushes, n);
    }
    first = g.shfl(first, 0);
    rest = g.shfl(rest, 0);
    served = g.shfl(served, 0);
    if (served & 0x100u) return rest + r < P.slots ? P.slots - 1u - (rest + r) : P.slots;
    return r < served ? first + r : rest + (r - served);
}

// Mark what is left of the block's chunks (whole block, after its last push).
__device__ inline void close_round(const TransportParams& P, const Round& R) {
    for (int k = 0; k < 2; ++k) {
        const uint32_t word = R.chunk[k];
        const unsigned int off = word & kOffMask;
        if (off >= kChunk) continue;
        if (threadIdx.x == 0) atomicAdd(&P.sched->dead[R.q_out[k]].v, kChunk - off);
        for (unsigned int i = off + threadIdx.x; i < kChunk; i += blockDim.x) {
            const unsigned int slot = (word >> kOffBits) * kChunk + i;
            if (slot < P.slots) P.q[R.q_out[k]][slot].d = make_uint4(kDeadMeta, 0u, 0u, 0u);
        }
    }
}

__device__ __forceinline__ const Slot* input_slot(const TransportParams& P, const Round& R, unsigned int i) {
    return P.q[R.q_in] + (i < R.n_bottom ? i : P.slots - 1u - (i - R.n_bottom));
}

// How a warp takes its share of the round's input: particles claimed R.claim at a
// time (one atomic, their slots prefetched into the L2) and handed to idle lanes.
struct Claim {
    unsigned int next = 0u, left = 0u;
    // The particle number of each lane that wants one (all lanes of the warp call).
    __device__ __forceinline__ unsigned int take(const TransportParams& P, const Round& R, bool want) {
        const unsigned int need = __ballot_sync(0xffffffffu, want);
        const unsigned int lane = threadIdx.x & 31u;
        const unsigned int cnt = (unsigned int)__popc(need);
        const unsigned int rank = (unsigned int)__popc(need & ((1u << lane) - 1u));
        unsigned int i = next + rank;
        if (cnt > left) {
            const unsigned int more = max(R.claim, cnt - left);
            unsigned int b = 0u;
            if (lane == 0u) b = atomicAdd(&P.sched->head[R.q_in].v, more);
            b = __shfl_sync(0xffffffffu, b, 0);
            if (lane < more && b + lane < R.n)
                asm volatile("prefetch.global.L2 [%0];" ::"l"(
                    __cvta_generic_to_global(input_slot(P, R, b + lane))));
            if (rank >= left) i = b + (rank - left);
            next = b + (cnt - left);
            left = more - (cnt - left);
        } else {
            next += cnt;
            left -= cnt;
        }
        return i;
    }
};

__device__ __forceinline__ void write_particle(const TransportParams& P, int qi, unsigned int idx, int kind,
                                               int beamlet, float e, float w, float x, float y, float z,
                                               float ux, float uy, float uz, const StreamId& sid) {
    if (idx >= P.slots) {
        atomicOr(&P.sched->flags, kFlagOverflow);
        return;
    }
    Slot* s = P.q[qi] + idx;
    s->a = make_float4(e, w, x, y);
    s->b = make_float4(z, ux, uy, uz);
    s->c = make_uint4(sid.id_lo, sid.id_hi, sid.tag, sid.ctr);
    s->d = make_uint4(pack_meta(kind, 0, beamlet), 0u, 0u, 0u);
}

__device__ __forceinline__ void queue_push(const TransportParams& P, Round& R, int k, int kind, int beamlet,
                                           float e, float w, float x, float y, float z, float ux, float uy,
                                           float uz, const StreamId& sid) {
    const unsigned int idx = claim_slot(P, R, k);
    write_particle(P, R.q_out[k], idx, kind, beamlet, e, w, x, y, z, ux, uy, uz, sid);
}

// ---- particle state ----------------------------------------------------------------
template <class R>
struct ParticleOf {
    float e, w, x, y, z, ux, uy, uz;
    uint32_t meta;  // as in a slot: kind, primary, beamlet in one register
    int steps;      // the host caps max_steps below 2^31
    R rng;
    __device__ __forceinline__ int kind() const { return (int)(meta & 3u); }
    __device__ __forceinline__ bool primary() const { return (meta & 4u) != 0u; }
    __device__ __forceinline__ int beamlet() const { return (int)(meta >> 3); }
};
using Particle = ParticleOf<Rng>;  // of the generator

// False for a dead slot.
template <class R>
__device__ __forceinline__ bool load_slot(const Slot* s, ParticleOf<R>& p) {
    const float4 a = s->a, b = s->b;
    const uint4 c = s->c, d = s->d;
    p.e = a.x; p.w = a.y; p.x = a.z; p.y = a.w;
    p.z = b.x; p.ux = b.y; p.uy = b.z; p.uz = b.w;
    p.meta = d.x;
    p.steps = (int)d.y;
    p.rng.load(StreamId{c.x, c.y, c.z, c.w});
    return d.x != kDeadMeta;
}

// A particle's whole state (phase space, kind, primary flag, beamlet, stream
// position, steps taken) in a slot: whoever loads it continues exactly there.
template <class R>
__device__ __forceinline__ void store_slot(Slot* s, const ParticleOf<R>& p) {
    const StreamId sid = p.rng.state();
    s->a = make_float4(p.e, p.w, p.x, p.y);
    s->b = make_float4(p.z, p.ux, p.uy, p.uz);
    s->c = make_uint4(sid.id_lo, sid.id_hi, sid.tag, sid.ctr);
    s->d = make_uint4(p.meta, (uint32_t)p.steps, 0u, 0u);
}

// Park an unfinished particle in output queue k for the next round.
template <class R>
__device__ __forceinline__ void queue_suspend(const TransportParams& P, Round& round, int k, const ParticleOf<R>& p) {
    const unsigned int idx = claim_slot(P, round, k);
    if (idx >= P.slots) atomicOr(&P.sched->flags, kFlagOverflow);
    else store_slot(P.q[round.q_out[k]] + idx, p);
}

// Copy `n` table entries into the block's shared memory (strided over the block).
template <typename T>
__device__ __forceinline__ void stage(T* dst, const T* src, int n) {
    for (int i = threadIdx.x; i < n; i += blockDim.x) dst[i] = __ldg(src + i);
}

// Vacuum flight to the grid for a particle born outside (photon.py:137-148);
// returns false (its energy escapes) when the flight misses the grid.
template <class R>
__device__ __forceinline__ bool enter_grid(const TransportParams& P, ParticleOf<R>& p) {
    if (point_inside(p.x, p.y, p.z, P.gi)) return true;
    float t = slab_entry_distance(p.x, p.y, p.z, p.ux, p.uy, p.uz, P.gi);
    if (t >= kInfinityCm) return false;
    t += kEntryNudge;
    p.x += t * p.ux;
    p.y += t * p.uy;
    p.z += t * p.uz;
    return point_inside(p.x, p.y, p.z, P.gi);
}

// The transmission of a user mask plane along the primary's full line
// (_MaskTransmission.factors, geometry/collimation.py:1041-1080; device twin
// kernels.py:2190-2244): zero for a ray parallel to the plane or crossing it
// outside the rectangle, else the bilinear value between pixel centres,
// clamped in the half-pixel border, in the incremental form that leaves a
// plateau of equal pixels exactly at their value.
__device__ inline float mask_transmission(const GenDesc& G, const Particle& p) {
    const float nx = G.muy * G.mvz - G.muz * G.mvy;
    const float ny = G.muz * G.mvx - G.mux * G.mvz;
    const float nz = G.mux * G.mvy - G.muy * G.mvx;
    const float den = p.ux * nx + p.uy * ny + p.uz * nz;
    if (den == 0.0f) return 0.0f;
    const float t = ((G.mcx - p.x) * nx + (G.mcy - p.y) * ny + (G.mcz - p.z) * nz) / den;
    const float ox = p.x + t * p.ux - G.mcx;
    const float oy = p.y + t * p.uy - G.mcy;
    const float oz = p.z + t * p.uz - G.mcz;
    const float u = ox * G.mux + oy * G.muy + oz * G.muz;
    const float v = ox * G.mvx + oy * G.mvy + oz * G.mvz;
    if (!(fabsf(u) <= 0.5f * G.mask_wu && fabsf(v) <= 0.5f * G.mask_wv)) return 0.0f;
    const int nu = G.mask_n_u, nv = G.mask_n_v;
    float pu = (u + 0.5f * G.mask_wu) / (G.mask_wu / (float)nu) - 0.5f;
    float pv = (v + 0.5f * G.mask_wv) / (G.mask_wv / (float)nv) - 0.5f;
    pu = fmaxf(0.0f, fminf(pu, (float)(nu - 1)));
    pv = fmaxf(0.0f, fminf(pv, (float)(nv - 1)));
    const int i0 = min((int)pu, max(nu - 2, 0));
    const int j0 = min((int)pv, max(nv - 2, 0));
    const int i1 = min(i0 + 1, nu - 1);
    const int j1 = min(j0 + 1, nv - 1);
    const float fu = pu - (float)i0, fv = pv - (float)j0;
    const float v00 = __ldg(G.mask + i0 * nv + j0), v10 = __ldg(G.mask + i1 * nv + j0);
    const float v01 = __ldg(G.mask + i0 * nv + j1), v11 = __ldg(G.mask + i1 * nv + j1);
    return v00 + fu * (v10 - v00) + fv * (v01 - v00) + fu * fv * (v11 - v10 - v01 + v00);
}

// Narrow-beam transmission of a collimated source (_StackTransmission.factors,
// geometry/collimation.py:927-985): exp(-sum_j mu_j(E) t_j), t_j the chord of
// the primary's full line through device j and mu_j that device's macroscopic
// total attenuation on its log-log table.  A ray trapped in a slab has an
// infinite chord and a zero transmission.
__device__ inline float stack_transmission(const GenDesc& G, const Particle& p) {
    const float x[3] = {p.x, p.y, p.z}, u[3] = {p.ux, p.uy, p.uz};
    float lp[3], ld[3];
    pmc_head::to_local(G.stack, x, u, lp, ld);
    float tau = 0.0f;
    for (int j = 0; j < G.stack.n; ++j) {
        const float t = pmc_head::device_len(G.stack, j, lp, ld, 0);
        if (t > 0.0f) tau += pmc_head::mu_at(G.stack_mu, G.stack_mu.log_total, j, p.e) * t;
    }
    return expf(-tau);
}

// ---- primary generation (kernels.py:1888-2401) -------------------------------------
// Maps primary t of the current wave (batches `batch` and up, one block each) to
// its batch, beamlet and history, seeds the history's stream, and samples the
// primary exactly as the host sources do
// (same uniforms, same order).  Returns the particle kind, or -1 when the
// source emits nothing for this history (a masked fan's zero transmission).
__device__ inline int generate_primary(const TransportParams& P, const GenDesc& G, int batch,
                                       unsigned long long t, Particle& p, long long& emitted) {
    // G is the device-resident descriptor, read field by field as needed.
    int local = 0;
    int map = 0;  // the wave's quanta map this primary's batch scores into
    if (G.wave_block) {
        map = (int)(t / G.wave_block);
        t -= (unsigned long long)map * G.wave_block;
        batch += map;
    }
    long long key;
    long long record;
    if (G.forward) {
        key = (long long)batch * G.per_batch_fwd + (long long)t;
        record = key;
    } else {
        int lo = 0, hi = G.group;  // largest local with pb_prefix[local] <= t
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if ((unsigned long long)__ldg(G.pb_prefix + mid) <= t) lo = mid;
            else hi = mid;
        }
        local = lo;
        const long long i = (long long)t - __ldg(G.pb_prefix + local);
        const long long r = (long long)batch * __ldg(G.per_batch + local) + i;
        const long long h = __ldg(G.hist_offset + local) + r;
        key = G.correlated ? r : h;
        record = h;
    }
    p.rng.k0 = P.seed_lo;
    p.rng.k1 = P.seed_hi;
    p.rng.id_lo = (uint32_t)((unsigned long long)key & 0xffffffffull);
    p.rng.id_hi = (uint32_t)((unsigned long long)key >> 32);
    p.rng.tag = 0u;
    p.rng.ctr = 0u;
    int kind = G.kind;
    p.steps = 0;
    p.w = 1.0f;
    if (G.type == 0) {  // pencil: no draws
        p.e = G.energy;
        p.x = G.px; p.y = G.py; p.z = G.pz;
        p.ux = G.dx; p.uy = G.dy; p.uz = G.dz;
    } else if (G.type == 1) {  // parallel field / beamlet lattice: two uniforms
        p.e = G.energy;
        p.x = __ldg(G.x_lo + local) + __ldg(G.x_ext + local) * p.rng.uniform();
        p.y = __ldg(G.y_lo + local) + __ldg(G.y_ext + local) * p.rng.uniform();
        p.z = G.z0;
        p.ux = 0.0f; p.uy = 0.0f; p.uz = 1.0f;
    } else if (G.type == 2) {  // divergent spectral fan: four uniforms
        const float u_bin = p.rng.uniform();
        const float u_within = p.rng.uniform();
        const float du = (p.rng.uniform() - 0.5f) * G.width_u;
        const float dv = (p.rng.uniform() - 0.5f) * G.width_v;
        int lo = 0, hi = G.n_bins;  // lower_bound: first k with cdf[k] >= u_bin
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (__ldg(G.cdf + mid) < u_bin) lo = mid + 1;
            else hi = mid;
        }
        const int k = min(lo, G.n_bins - 1);
        const float e_lo = __ldg(G.edges + k);
        p.e = e_lo + (__ldg(G.edges + k + 1) - e_lo) * u_within;
        const float dx = __ldg(G.cx + local) + du * G.uax + dv * G.vax - G.fx;
        const float dy = __ldg(G.cy + local) + du * G.uay + dv * G.vay - G.fy;
        const float dz = __ldg(G.cz + local) + du * G.uaz + dv * G.vaz - G.fz;
        const float inv = 1.0f / sqrtf(dx * dx + dy * dy + dz * dz);
        p.x = G.fx; p.y = G.fy; p.z = G.fz;
        p.ux = dx * inv; p.uy = dy * inv; p.uz = dz * inv;
    } else if (G.type == 4) {  // per-beamlet record (CompositeBeamletSource.emit for mixtures)
        const BeamletRec* r = G.recs + (long long)local * G.n_comp;
        if (G.n_comp > 1) {  // one uniform: the first component whose cdf reaches it
            const float u = p.rng.uniform();
            int lo = 0, hi = G.n_comp;
            while (lo < hi) {
                const int mid = (lo + hi) >> 1;
                if (__ldg(G.comp_cdf + mid) < u) lo = mid + 1;
                else hi = mid;
            }
            r += min(lo, G.n_comp - 1);
        }
        const float4 a = __ldg(&r->a), b = __ldg(&r->b);
        const float4 d = __ldg(&r->d);
        const int bits = __float_as_int(d.w);
        kind = kPhoton;
        if ((bits & 1) == 0) {  // lattice rectangle: two uniforms
            p.e = b.y;
            p.x = a.x + a.y * p.rng.uniform();
            p.y = a.z + a.w * p.rng.uniform();
            p.z = b.x;
            p.ux = 0.0f; p.uy = 0.0f; p.uz = 1.0f;
        } else {  // divergent fan through the aperture: four uniforms
            const float4 c = __ldg(&r->c);
            const int first = __float_as_int(c.w);
            const int n_bins = bits >> 1;
            const float u_bin = p.rng.uniform();
            const float u_within = p.rng.uniform();
            const float du = (p.rng.uniform() - 0.5f) * a.w;
            const float dv = (p.rng.uniform() - 0.5f) * b.w;
            int lo = 0, hi = n_bins;
            while (lo < hi) {
                const int mid = (lo + hi) >> 1;
                if (__ldg(G.cdf + first + mid) < u_bin) lo = mid + 1;
                else hi = mid;
            }
            const int k = first + min(lo, n_bins - 1);
            const float e_lo = __ldg(G.edges + k);
            p.e = e_lo + (__ldg(G.edges + k + 1) - e_lo) * u_within;
            const float dx = b.x + du * c.x + dv * d.x - a.x;
            const float dy = b.y + du * c.y + dv * d.y - a.y;
            const float dz = b.z + du * c.z + dv * d.z - a.z;
            const float inv = 1.0f / sqrtf(dx * dx + dy * dy + dz * dz);
            p.x = a.x; p.y = a.y; p.z = a.z;
            p.ux = dx * inv; p.uy = dy * inv; p.uz = dz * inv;
        }
    } else {  // host-sampled record: the run's history, or the batch block's slot t (Dij);
              // resident phase space: a record drawn by the history's own stream
        long long ri = G.forward ? record : (long long)t;
        if (G.type == 5) {
            const unsigned long long r =
                ((unsigned long long)p.rng.next_u32() << 32) | (unsigned long long)p.rng.next_u32();
            ri = (long long)__umul64hi(r, (unsigned long long)G.n_records);
        }
        kind = G.up_kind ? __ldg(G.up_kind + ri) : kPhoton;
        p.e = __ldg(G.up_energy + ri);
        p.w = __ldg(G.up_weight + ri);
        p.x = __ldg(G.up_pos + 3 * ri);
        p.y = __ldg(G.up_pos + 3 * ri + 1);
        p.z = __ldg(G.up_pos + 3 * ri + 2);
        p.ux = __ldg(G.up_dir + 3 * ri);
        p.uy = __ldg(G.up_dir + 3 * ri + 1);
        p.uz = __ldg(G.up_dir + 3 * ri + 2);
    }
    p.meta = pack_meta(kind, 1, map * G.group + local);
    if (G.type != 3 && G.type != 5) {  // host records carry their own weights
        // a zero weight emits nothing; the history still counts in the batch mean
        if (G.masked) p.w *= mask_transmission(G, p);
        if (G.stacked && p.w != 0.0f) p.w *= stack_transmission(G, p);
        if (p.w == 0.0f) return -1;
    }
    if (G.book_emitted) {
        const float latent = kind == kPositron ? 2.0f * kElectronMass : 0.0f;
        emitted += quantize_signed(p.w * (p.e + latent));
    }
    return kind;
}

// ---- annihilation at rest (transport/particles.py:75, kernels.py:675) ------------
// (output queue 1 is the photon queue of both kernels)
template <bool kPlain, class R, class Sink>
__device__ __forceinline__ void annihilate_at_rest(const TransportParams& P, BlockBooks& B, ParticleOf<R>& p,
                                                   int voxel, Round& round, float factor, Sink& sink) {
    if (P.pcut >= kElectronMass) {
        deposit<kPlain>(P, B, p.beamlet(), p.x, p.y, p.z, voxel, p.w * 2.0f * kElectronMass, factor, sink);
        return;
    }
    float ax, ay, az;
    p.rng.reserve(2);
    sample_isotropic_direction(p.rng, ax, ay, az);
#pragma unroll 1
    for (int k = 0; k < 2; ++k) {  // two photons back to back
        p.rng.reserve(3);
        const StreamId sid = p.rng.spawn();
        queue_push(P, round, 1, kPhoton, p.beamlet(), kElectronMass, p.w, p.x, p.y, p.z, ax, ay, az, sid);
        ax = -ax;
        ay = -ay;
        az = -az;
    }
}

__device__ __forceinline__ void retire_queue(Sched* S, int qi) {
    S->bottom[qi].v = S->top[qi].v = S->head[qi].v = S->dead[qi].v = 0u;
}

// Set the next admission window's slots aside at the bottom of the queue its
// primaries enter (nothing else is pushed until they are written).
__device__ __forceinline__ void open_window(Sched* S, int window_el) {
    unsigned int* bottom = &S->bottom[window_el ? 2 + S->e_in : S->p_in].v;
    const unsigned int base = __ldcg(bottom);
    S->window_base = base;
    *bottom = base + round_to_chunk(S->limit - S->cursor);
}

// ---- last-block scheduler steps ------------------------------------------------------
__device__ inline bool last_block_arrives(Sched* S) {
    __shared__ bool last;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        const unsigned int done = atomicAdd(&S->blocks_done, 1u);
        last = (done == gridDim.x - 1);
    }
    __syncthreads();
    return last;
}

__device__ inline void flush_books(const TransportParams& P, BlockBooks& B) {
    __syncthreads();
    if (threadIdx.x == 0) {
        Counters* C = P.counters;
        if (B.flights) atomicAdd(&C->flights, B.flights);
        if (B.interactions) atomicAdd(&C->interactions, B.interactions);
        if (B.substeps) atomicAdd(&C->substeps, B.substeps);
        if (B.deposits) atomicAdd(&C->deposits, B.deposits);
        if (B.pushes) atomicAdd(&C->pushes, B.pushes);
        if (B.primaries) atomicAdd(&C->primaries, B.primaries);
        book_add(&C->escaped, B.escaped);
        book_add(&C->unscored, B.unscored);
        book_add(&C->deposited, B.deposited);
        book_add(&C->emitted, B.emitted);
        book_add(&C->violations, B.violations);
    }
}

__device__ __forceinline__ void init_books(BlockBooks& B) {
    if (threadIdx.x == 0) {
        B.flights = B.interactions = B.substeps = B.deposits = B.pushes = B.primaries = B.dead = 0ull;
        B.escaped = B.unscored = B.deposited = B.emitted = B.violations = 0ll;
    }
    __syncthreads();
}

__device__ __forceinline__ void block_sum_add(unsigned long long* dst, unsigned long long v) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    if ((threadIdx.x & 31) == 0 && v) atomicAdd(dst, v);
}

// ---- the photon kernel ---------------------------------------------------------------
constexpr int kPhotonThreads = 256;  // the largest block of the photon kernel

// One lane transports one photon to termination (Woodcock tracking), then takes
// the round's next queued photon.
// kSmem: the channel rows of every material and the majorant row are staged in
// the block's shared memory (dynamic, n_materials * n_points * 16 + n_points * 4
// bytes) instead of being read through L1.
// kMinBlocks: resident blocks of 256 per SM the register allocation targets (3:
// 72 registers, 4: 64, no spills either way).
// kPlain: dose to medium on the transport grid itself, whole-substep deposits, no
// Compton splitting, fewer than 2^31 voxels (plain_scoring): a deposit's bin is the
// voxel already at hand.
template <bool kSmem, int kMinBlocks, bool kPlain>
__global__ void __launch_bounds__(kPhotonThreads, kMinBlocks) photon_kernel(const __grid_constant__ TransportParams P) {
    __shared__ BlockBooks B;
    __shared__ uint32_t ring[kRingWords * kPhotonThreads];
    extern __shared__ __align__(16) unsigned char pmc_smem[];
    const float4* tab_ch = P.tab.ch;
    const float* tab_maj = P.tab.maj;
    if constexpr (kSmem) {
        const int n = P.tab.n_materials * P.tab.n_points;
        float4* sch = reinterpret_cast<float4*>(pmc_smem);
        float* smaj = reinterpret_cast<float*>(sch + n);
        stage(sch, P.tab.ch, n);
        stage(smaj, P.tab.maj, P.tab.n_points);
        tab_ch = sch;
        tab_maj = smaj;
    }
    Sched* S = P.sched;
    __shared__ Round rd;  // pushes electrons (0) and, rarely, photons (1)
    if (threadIdx.x == 0) open_round(P, rd, S->p_in, 2 + S->e_in, S->p_in ^ 1, 1u);
    init_books(B);  // its barrier also publishes the round and the staged tables
    const Tables& T = P.tab;
    const float pcut = P.pcut, ecut = P.ecut;

    Claim input;
    unsigned int n_flight = 0, n_inter = 0;  // per lane and launch
    DirectSink dep;
    ParticleOf<RingRng<kPhotonThreads, true>> p;
    p.rng.keys = &P.keys;
    p.rng.ring = ring + threadIdx.x;
    long long escaped = 0;  // most photons end that way: summed per lane, booked once
    auto leave = [&](float amount) { escaped += quantize_signed(amount); };
    bool active = false, exhausted = false;
    int tail = -1;  // turns since the warp found the round dry
    float e_tab = -1.0f, maj = 0.0f;
    LogIdx li{0, 0.0f};
    int mat_tab = -1;
    float4 ch = make_float4(0.f, 0.f, 0.f, 0.f);

    for (unsigned int it = 0;; ++it) {
        if ((it & 255u) == 0u) {
            if (__any_sync(0xffffffffu, (*(volatile int*)&S->flags) & (kFlagOverflow | kFlagStepCap)))
                break;
        }
        const bool want = !active && !exhausted;  // the round's photons: secondaries, primaries, parked
        if (__any_sync(0xffffffffu, want)) {
            const unsigned int i = input.take(P, rd, want);
            if (want) {
                if (i < rd.n) {
                    if (load_slot(input_slot(P, rd, i), p)) {
                        active = enter_grid(P, p);
                        if (!active) leave(p.w * p.e);
                    }
                    e_tab = -1.0f;
                } else {
                    exhausted = true;
                }
            }
        }
        if (!__any_sync(0xffffffffu, active || !exhausted)) break;
        // Once the round's input has run dry, a photon that still needs more than
        // tail_steps flights is parked for the next round instead of holding its
        // warp (and its block's barrier) while every other lane idles.
        if (tail >= 0 || __any_sync(0xffffffffu, exhausted)) ++tail;
        if (!active) continue;
        if (tail >= P.tail_steps) {
            queue_suspend(P, rd, 1, p);
            active = false;
            continue;
        }

        // ---- one Woodcock flight (photon.py:150-181) ----
        if (++p.steps > P.max_steps) {
            atomicOr(&S->flags, kFlagStepCap);
            leave(p.w * p.e);
            active = false;
            continue;
        }
        p.rng.top_up();  // path, acceptance, channel
        if (p.e != e_tab) {
            li = log_index(p.e, T.p_log_min, T.p_inv_dlog, T.n_points);
            maj = lerp1<kSmem>(tab_maj, li);
            e_tab = p.e;
            mat_tab = -1;
        }
        ++n_flight;
        const float step = sample_path_length(maj, p.rng);
        p.x += step * p.ux;
        p.y += step * p.uy;
        p.z += step * p.uz;
        if (!point_inside(p.x, p.y, p.z, P.gi)) {
            leave(p.w * p.e);
            active = false;
            continue;
        }
        const BinOf<kPlain> flat = voxel_of<kPlain>(p.x, p.y, p.z, P.gi);
        const float2 vx = __ldg(P.vox + flat);
        const int voxel = kPlain ? (int)flat : 0;
        const float rho = vx.x;
        const int mat = __float_as_int(vx.y);
        if (mat != mat_tab) {
            ch = lerp4<kSmem>(tab_ch + (long long)mat * T.n_points, li);
            mat_tab = mat;
        }
        const float mc = rho * ch.x, mp = rho * ch.y, mpa = rho * ch.z, mr = rho * ch.w;
        const float mu_real = mc + mp + mpa + mr;
        if (mu_real > maj * (1.0f + 1.0e-9f)) {
            book_add(&B.violations, 1);
            leave(p.w * p.e);
            active = false;
            continue;
        }
        if (p.rng.uniform() * maj >= mu_real) continue;  // delta scattering
        ++n_inter;
        const int process = select_photon_process(mc, mp, mpa, mr, p.rng);
        auto put = [&](float amount, float energy) {  // local deposit of an electron of that energy
            deposit<kPlain>(P, B, p.beamlet(), p.x, p.y, p.z, voxel, amount,
                            kPlain ? 1.0f : spr_factor(P, energy, mat), dep);
        };

        if (process == 3) {  // coherent
            const float c = sample_coherent_cos_theta(T, mat, p.e, p.rng);
            p.rng.reserve(1);
            const float phi = kTwoPi * p.rng.uniform();
            rotate_direction(p.ux, p.uy, p.uz, c, phi);
            continue;
        }
        if (!kPlain && process == 0 && P.split_n > 1 && p.primary()) {
            // Compton splitting of a source photon (photon.py:190-224): N
            // copies of weight w/N, each pushed as a non-primary photon.
            const float split_w = p.w / (float)P.split_n;
            for (int k = 0; k < P.split_n; ++k) {
                const float ratio = sample_compton_energy_ratio(p.e, p.rng);
                const float recoil = p.e * (1.0f - ratio);
                p.rng.reserve(4);
                const float phi = kTwoPi * p.rng.uniform();
                if (P.transport_electrons && recoil > ecut) {
                    float ex = p.ux, ey = p.uy, ez = p.uz;
                    rotate_direction(ex, ey, ez, compton_electron_cos_theta(p.e, ratio), phi + kPi);
                    const StreamId sid = p.rng.spawn();
                    queue_push(P, rd, 0, kElectron, p.beamlet(), recoil, split_w, p.x, p.y, p.z, ex, ey, ez, sid);
                } else {
                    put(split_w * recoil, recoil);
                }
                float gx = p.ux, gy = p.uy, gz = p.uz;
                rotate_direction(gx, gy, gz, compton_cos_theta(p.e, ratio), phi);
                const float es = p.e * ratio;
                if (es <= pcut) {
                    put(split_w * es, es);
                    continue;
                }
                float cw = split_w;
                bool keep = true;
                p.rng.reserve(4);
                if (es < kRouletteMeV && cw < kRouletteWeightCap) {
                    const float nw = roulette_weight(cw, kRouletteSurvival, p.rng);
                    leave((cw - nw) * es);
                    if (nw == 0.0f) keep = false;
                    else cw = nw;
                }
                if (keep) {
                    const StreamId sid = p.rng.spawn();
                    queue_push(P, rd, 1, kPhoton, p.beamlet(), es, cw, p.x, p.y, p.z, gx, gy, gz, sid);
                }
            }
            active = false;
            continue;
        }

        // Compton, photoelectric and pair events each set one electron in motion
        // (electron energy ee, direction ex, ey, ez): found per process, then
        // pushed or deposited in one place for all of them.
        float ratio = 0.0f, phi = 0.0f, kinetic = 0.0f, fraction = 0.0f;
        float ee, ex = p.ux, ey = p.uy, ez = p.uz;
        if (process == 0) {
            ratio = sample_compton_energy_ratio(p.e, p.rng);
            ee = p.e * (1.0f - ratio);
        } else if (process == 1) {  // photoelectric: forward, no fluorescence
            ee = p.e;
        } else {
            kinetic = p.e - 2.0f * kElectronMass;
            ee = kinetic;  // without electron transport the pair's energy stays here
        }
        p.rng.reserve(4);
        if (process == 0) {
            phi = kTwoPi * p.rng.uniform();
        } else if (process == 2 && P.transport_electrons) {
            fraction = p.rng.uniform();
            ee = fraction * kinetic;
        }
        if (P.transport_electrons && ee > ecut) {
            if (process == 0)
                rotate_direction(ex, ey, ez, compton_electron_cos_theta(p.e, ratio), phi + kPi);
            const StreamId sid = p.rng.spawn();
            queue_push(P, rd, 0, kElectron, p.beamlet(), ee, p.w, p.x, p.y, p.z, ex, ey, ez, sid);
        } else {
            put(p.w * ee, ee);
        }

        if (process == 0) {
            rotate_direction(p.ux, p.uy, p.uz, compton_cos_theta(p.e, ratio), phi);
            p.e *= ratio;
            if (p.e <= pcut) {
                put(p.w * p.e, p.e);
                active = false;
                continue;
            }
            if (p.e < kRouletteMeV && p.w < kRouletteWeightCap) {
                p.rng.reserve(1);
                const float nw = roulette_weight(p.w, kRouletteSurvival, p.rng);
                leave((p.w - nw) * p.e);
                if (nw == 0.0f) {
                    active = false;
                    continue;
                }
                p.w = nw;
            }
            continue;
        }
        if (process == 2) {  // pair production: the positron
            const float share_p = (1.0f - fraction) * kinetic;
            if (P.transport_electrons && share_p > ecut) {
                p.rng.reserve(3);
                const StreamId sid = p.rng.spawn();
                queue_push(P, rd, 0, kPositron, p.beamlet(), share_p, p.w, p.x, p.y, p.z, p.ux, p.uy, p.uz, sid);
            } else {
                if (P.transport_electrons) put(p.w * share_p, share_p);
                annihilate_at_rest<kPlain>(P, B, p, voxel, rd,
                                           kPlain ? 1.0f : spr_factor(P, kElectronMass, mat), dep);
            }
        }
        active = false;
    }

    __syncthreads();
    close_round(P, rd);
    if (threadIdx.x == 0) B.pushes += rd.pushes;
    block_sum_add(reinterpret_cast<unsigned long long*>(&B.escaped), (unsigned long long)escaped);
    block_sum_add(&B.flights, n_flight);
    block_sum_add(&B.interactions, n_inter);
    block_sum_add(&B.deposits, dep.n);
    flush_books(P, B);

    // The last block retires the consumed photon queue; the round's admission
    // window has been generated.
    if (last_block_arrives(S) && threadIdx.x == 0) {
        retire_queue(S, rd.q_in);
        S->p_in = rd.q_out[1];
        S->cursor = S->limit;
        S->blocks_done = 0u;
        __threadfence();
    }
}

// ---- the primary generator ---------------------------------------------------------
// The round's admission window [cursor, limit) of the wave, one thread
// per primary (kernels.py:1888-2401): sampled at full warp width, flown
// through vacuum to the grid, then queued with its stream position.  The slots
// are set aside by the scheduler, primary t in slot window_base + (t - cursor)
// (no atomics) of the photon queue, behind the secondaries already there, or of
// the electron queue for a charged source; a primary that is not to be
// transported there leaves its slot dead, a charged one of a mixed source goes to
// the electron queue.
__global__ void __launch_bounds__(256) generate_kernel(const __grid_constant__ TransportParams P) {
    __shared__ BlockBooks B;
    init_books(B);
    Sched* S = P.sched;
    const unsigned long long cursor = S->cursor, limit = S->limit;
    const int q_ph = S->p_in, q_el = 2 + S->e_in;
    const int q_win = P.window_el ? q_el : q_ph;
    const unsigned int base = S->window_base;
    const int batch = S->batch;
    const GenDesc& G = *P.gen;
    unsigned int n_push = 0, n_prim = 0, n_dead = 0;
    long long emitted = 0, escaped = 0;  // per thread, booked once per warp
    const unsigned long long stride = (unsigned long long)gridDim.x * blockDim.x;
    const unsigned int window = round_to_chunk(limit - cursor);
    for (unsigned long long k = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; k < window; k += stride) {
        Particle p;
        const unsigned int slot = base + (unsigned int)k;
        bool queued = false;
        if (cursor + k < limit) {
            ++n_prim;
            const int kind = generate_primary(P, G, batch, cursor + k, p, emitted);
            if (kind >= 0 && P.window_el) {
                queued = true;  // (it enters the grid in the electron kernel)
            } else if (kind == kPhoton) {
                queued = enter_grid(P, p);
                if (!queued) escaped += quantize_signed(p.w * p.e);
            } else if (kind > 0) {
                write_particle(P, q_el, single_slot(P, q_el), kind, p.beamlet(), p.e, p.w, p.x, p.y, p.z, p.ux,
                               p.uy, p.uz, p.rng.state());
                ++n_push;
            }
        }
        n_push += queued ? 1u : 0u;
        n_dead += queued ? 0u : 1u;
        if (slot >= P.slots) {
            atomicOr(&S->flags, kFlagOverflow);
        } else if (queued) {
            store_slot(P.q[q_win] + slot, p);
        } else {
            P.q[q_win][slot].d = make_uint4(kDeadMeta, 0u, 0u, 0u);
        }
    }
    block_sum_add(&B.pushes, n_push);
    block_sum_add(&B.primaries, n_prim);
    block_sum_add(&B.dead, n_dead);
    block_sum_add(reinterpret_cast<unsigned long long*>(&B.emitted), (unsigned long long)emitted);
    block_sum_add(reinterpret_cast<unsigned long long*>(&B.escaped), (unsigned long long)escaped);
    flush_books(P, B);
    if (threadIdx.x == 0 && B.dead) atomicAdd(&S->dead[q_win].v, (unsigned int)B.dead);
}

// Annihilation energy a positron still carries (2 m c^2), booked with it on escape.
template <class R>
__device__ __forceinline__ float rest_energy(const ParticleOf<R>& p) {
    return p.kind() == kPositron ? 2.0f * kElectronMass : 0.0f;
}

// ---- the electron kernel -------------------------------------------------------------
// What bounds both transport kernels: instruction issue with half the lanes
// active, then the latency of the voxel and queue gathers, not HBM.  On a
// 100-column 128^3 Dij (1.9e7 histories, 1.7e8 substeps, 7.8e7 flights), electron and
// photon kernel: 17.5 and 13.6 ms with a Philox block per lane in registers, one
// scoring path and single queue slots; 12.4 and 12.1 with the ring in shared memory, the
// plain scoring path and the terminal step folded into the refill; 10.5 and 5.3 with
// chunked slots and claims; 9.7 and 4.9 with blocks of 384 and the round keys at hand.
constexpr int kElectronThreads = 384;  // the largest block of the electron kernel

// One lane runs one electron or positron to ECUT (Class II condensed history,
// electron.py:345-481); delta rays go to the next round's electron queue,
// bremsstrahlung and annihilation photons to the next photon round.
// kSmem: the (csda range, moller, restricted range, radiative stopping) and
// (scattering power, log eta) rows of every material are staged in the block's
// shared memory (n_materials * n_points * 24 bytes); the inverse-range row
// (one read per substep) stays on the L1 path.
// kMinBlocks: resident blocks of 256 threads per SM the register allocation
// targets: 3 (85 registers; by default launched as two blocks of 384, which stage
// the tables twice per SM instead of three times) or 4 (64, with spills: 10.0 ms
// against 9.8 on the 100-column 128^3 Dij, and the longest electron of a small
// round takes longer: 0.35 against 0.30 ms on a 16^3 run).
// kPlain: as for the photon kernel.
template <bool kSmem, int kMinBlocks, bool kPlain>
__global__ void __launch_bounds__(kMinBlocks == 3 ? kElectronThreads : 256, kMinBlocks == 3 ? 2 : kMinBlocks)
electron_kernel(const __grid_constant__ TransportParams P) {
    __shared__ BlockBooks B;
    __shared__ uint32_t ring[kRingWords * kElectronThreads];
    extern __shared__ __align__(16) unsigned char pmc_smem[];
    const float4* tab_ea = P.tab.ea;
    const float2* tab_eb = P.tab.eb;
    if constexpr (kSmem) {
        const int n = P.tab.n_materials * P.tab.n_points;
        float4* sea = reinterpret_cast<float4*>(pmc_smem);
        float2* seb = reinterpret_cast<float2*>(sea + n);
        stage(sea, P.tab.ea, n);
        stage(seb, P.tab.eb, n);
        tab_ea = sea;
        tab_eb = seb;
    }
    Sched* S = P.sched;
    __shared__ Round rd;  // pushes the next round's electrons (0) and photons (1)
    if (threadIdx.x == 0) open_round(P, rd, 2 + S->e_in, 2 + (S->e_in ^ 1), S->p_in, 3u);
    init_books(B);  // its barrier also publishes the round and the staged tables
    const Tables& T = P.tab;
    const float pcut = P.pcut, ecut = P.ecut;

    Claim input;
    unsigned int n_sub = 0;  // per lane and launch
    HeldSink<BinOf<kPlain>> dep;
    ParticleOf<RingRng<kElectronThreads, false>> p;
    p.meta = 0u;
    p.rng.k0 = P.seed_lo;
    p.rng.k1 = P.seed_hi;
    p.rng.ring = ring + threadIdx.x;
    bool active = false, exhausted = false;
    int tail = -1;  // turns since the warp found the round dry

    for (unsigned int it = 0;; ++it) {
        if ((it & 255u) == 0u) {
            if (__any_sync(0xffffffffu, (*(volatile int*)&S->flags) & (kFlagOverflow | kFlagStepCap)))
                break;
        }
        // A particle that came to rest deposits and its lane takes the next one in
        // the same turn of the loop, so that no lane sits out a substep in between
        // (an electron lives 4.5 substeps on average).
        if (active && p.e <= ecut) {  // terminal: local deposit (electron.py:347-365)
            if (++p.steps > P.max_steps) {
                atomicOr(&S->flags, kFlagStepCap);
                escape(B, p.w * (p.e + rest_energy(p)));
            } else {
                const BinOf<kPlain> flat = voxel_of<kPlain>(p.x, p.y, p.z, P.gi);
                const int voxel = kPlain ? (int)flat : 0;
                const int tm = kPlain ? 0 : __float_as_int(__ldg(P.vox + flat).y);
                deposit<kPlain>(P, B, p.beamlet(), p.x, p.y, p.z, voxel, p.w * p.e,
                                kPlain ? 1.0f : spr_factor(P, p.e, tm), dep);
                if (p.kind() == kPositron)
                    annihilate_at_rest<kPlain>(P, B, p, voxel, rd,
                                               kPlain ? 1.0f : spr_factor(P, kElectronMass, tm), dep);
            }
            active = false;
        }
        if (!active) dep.release(P, p.beamlet());  // the finished particle's last held deposit
        const bool want = !active && !exhausted;
        if (__any_sync(0xffffffffu, want)) {
            const unsigned int i = input.take(P, rd, want);
            if (want) {
                if (i < rd.n) {
                    if (load_slot(input_slot(P, rd, i), p)) {
                        active = enter_grid(P, p);
                        if (!active) escape(B, p.w * (p.e + rest_energy(p)));
                    }
                } else {
                    exhausted = true;
                }
            }
        }
        if (!__any_sync(0xffffffffu, active || !exhausted)) break;
        if (tail >= 0 || __any_sync(0xffffffffu, exhausted)) ++tail;
        if (!active || p.e <= ecut) continue;
        // Park a particle that outlives the round's input by tail_steps substeps
        // (its held deposit is released at the top of the next iteration).
        if (tail >= P.tail_steps) {
            queue_suspend(P, rd, 0, p);
            active = false;
            continue;
        }

        if (++p.steps > P.max_steps) {
            atomicOr(&S->flags, kFlagStepCap);
            escape(B, p.w * (p.e + rest_energy(p)));
            active = false;
            continue;
        }
        ++n_sub;
        p.rng.fill_both();  // a substep's five draws: path, brems, hinge point, angle, azimuth
        const float2 vx = __ldg(P.vox + voxel_of<kPlain>(p.x, p.y, p.z, P.gi));
        const float rho = vx.x;
        const int mat = __float_as_int(vx.y);
        const long long row = (long long)mat * T.n_points;

        // --- substep length ---
        const LogIdx le = log_index(p.e, T.e_log_min, T.e_inv_dlog, T.n_points);
        const float4 A = lerp4<kSmem>(tab_ea + row, le);  // csda, moller, restricted range, radiative
        const float range_cm = A.x / rho;
        float s_max = P.step_fraction * range_cm;
        if (!P.msc_gs) {
            const float tp = lerp2<kSmem>(tab_eb + row, le).x;
            s_max = fminf(s_max, kHingeTheta2Max / (tp * rho));
        }
        const float s_boundary =
            distance_to_voxel_boundary(p.x, p.y, p.z, p.ux, p.uy, p.uz, P.gi) + kBoundaryNudge;
        const float s_geometry = fminf(s_max, s_boundary);
        const float sigma_moller = rho * A.y;
        float s = s_geometry;
        bool moller_pending = false;
        if (sigma_moller > 0.0f) {
            const float s_int = sample_path_length(sigma_moller, p.rng);
            if (s_int <= s_geometry) {
                s = s_int;
                moller_pending = true;
            }
        }
        // --- continuous loss, exact DPM range map ---
        const float available = A.z;
        float de;
        if (rho * s >= available) {
            s = available / rho;
            de = p.e - ecut;
            moller_pending = false;
        } else {
            const LogIdx lr = log_index(available - rho * s, T.r_log_min, T.r_inv_dlog, T.n_points);
            float e_end = lerp1(T.er + row, lr);
            e_end = fminf(fmaxf(e_end, ecut), p.e);
            de = p.e - e_end;
        }
        float emit_p, local_brems;
        brems_step_parameters(p.e, A.w, rho, s, pcut, emit_p, local_brems);
        const float continuous = de + local_brems;
        const bool emit_brems = p.rng.uniform() < emit_p;
        const float factor = kPlain ? 1.0f : spr_factor(P, p.e, mat);

        // --- random hinge: move, deflect, move ---
        const float s1 = p.rng.uniform() * s;
        const float s2 = s - s1;
        float d1 = 0.0f;
        if (s > 0.0f) d1 = continuous * (s1 / s);
        const float d2 = continuous - d1;

        deposit_spread<kPlain>(P, B, p.beamlet(), p.x, p.y, p.z, p.ux, p.uy, p.uz, s1, p.w * d1, factor, dep);
        p.e -= d1;
        p.x += p.ux * s1;
        p.y += p.uy * s1;
        p.z += p.uz * s1;
        if (!point_inside(p.x, p.y, p.z, P.gi)) {
            escape(B, p.w * (p.e + rest_energy(p)));
            active = false;
            continue;
        }
        const LogIdx lh = log_index(p.e, T.e_log_min, T.e_inv_dlog, T.n_points);
        const float2 Bh = lerp2<kSmem>(tab_eb + row, lh);  // scattering power, log eta
        const float ms = Bh.x * rho * s;
        float cos_hinge;
        if (P.msc_gs) {
            const float fx = Bh.y * T.gs_bins_per_log;
            const float fy = logf(fmaxf(ms, kGsThetaMin2)) * T.gs_bins_per_log;
            cos_hinge = sample_gs_cos_theta(T, fx, fy, ms, p.rng);
        } else {
            cos_hinge = sample_hinge_cos_theta(ms, p.rng);
        }
        const float phi = kTwoPi * p.rng.uniform();
        rotate_direction(p.ux, p.uy, p.uz, cos_hinge, phi);

        if (emit_brems && p.e > pcut) {
            p.rng.reserve(2);
            float k = sample_brems_energy(p.e, pcut, p.rng);
            k = fminf(k, p.e - d2);
            if (k > pcut) {
                float pw = p.w;
                if (k < kRouletteMeV && p.w < kRouletteWeightCap) {
                    pw = roulette_weight(p.w, kRouletteSurvival, p.rng);
                    escape(B, (p.w - pw) * k);
                }
                if (pw > 0.0f) {
                    p.rng.reserve(3);
                    const StreamId sid = p.rng.spawn();
                    queue_push(P, rd, 1, kPhoton, p.beamlet(), k, pw, p.x, p.y, p.z, p.ux, p.uy, p.uz, sid);
                }
            } else {
                deposit_or_escape<kPlain>(P, B, p.beamlet(), p.x, p.y, p.z, p.w * k,
                                          kPlain ? 1.0f : spr_factor(P, k, mat), dep);
            }
            p.e -= k;
        }

        deposit_spread<kPlain>(P, B, p.beamlet(), p.x, p.y, p.z, p.ux, p.uy, p.uz, s2, p.w * d2, factor, dep);
        p.e -= d2;
        p.x += p.ux * s2;
        p.y += p.uy * s2;
        p.z += p.uz * s2;
        if (!point_inside(p.x, p.y, p.z, P.gi)) {
            escape(B, p.w * (p.e + rest_energy(p)));
            active = false;
            continue;
        }

        // --- discrete Moller event at the end of the substep ---
        if (moller_pending && p.e > 2.0f * ecut) {
            const float w = sample_moller_delta_energy(p.e, ecut, p.rng);
            float cd, cp;
            moller_direction_cosines(p.e, w, cd, cp);
            p.rng.reserve(4);
            const float mphi = kTwoPi * p.rng.uniform();
            float dx = p.ux, dy = p.uy, dz = p.uz;
            rotate_direction(dx, dy, dz, cd, mphi);
            const StreamId sid = p.rng.spawn();
            queue_push(P, rd, 0, kElectron, p.beamlet(), w, p.w, p.x, p.y, p.z, dx, dy, dz, sid);
            rotate_direction(p.ux, p.uy, p.uz, cp, mphi + kPi);
            p.e -= w;
        }
    }

    dep.release(P, p.beamlet());
    __syncthreads();
    close_round(P, rd);
    if (threadIdx.x == 0) B.pushes += rd.pushes;
    block_sum_add(&B.substeps, n_sub);
    block_sum_add(&B.deposits, dep.n);
    flush_books(P, B);

    // The last block retires the consumed electron queue, opens the next
    // admission window and publishes whether any work is left.
    if (last_block_arrives(S) && threadIdx.x == 0) {
        retire_queue(S, rd.q_in);
        S->e_in = rd.q_out[0] - 2;
        S->rounds += 1;
        S->total_rounds += 1;
        const unsigned long long next_limit = S->cursor + S->budget;
        S->limit = next_limit < S->block_end ? next_limit : S->block_end;
        // particles queued, beside the dead slots
        auto queued = [S](int qi) {
            return __ldcg(&S->bottom[qi].v) + __ldcg(&S->top[qi].v) > __ldcg(&S->dead[qi].v);
        };
        const bool work = S->cursor < S->block_end || queued(S->p_in) || queued(S->e_in + 2);
        open_window(S, P.window_el);
        int remaining = work ? 1 : 0;
        if (S->flags & (kFlagOverflow | kFlagStepCap)) remaining = 0;
        if (remaining && S->rounds >= S->max_rounds) {
            S->flags |= kFlagRoundCap;
            remaining = 0;
        }
        S->remaining = remaining;
        S->blocks_done = 0u;
        __threadfence();
        if (S->cond_handle != 0ull)
            cudaGraphSetConditional((cudaGraphConditionalHandle)S->cond_handle,
                                    (unsigned int)remaining);
    }
}

}  // namespace pmc
