// denoise_ws.cuh — the 3x3x3 convolution as a warp-specialized pipeline on the
// 5th-generation tensor cores, included by denoise.cu after denoise_umma.cuh.
//
// The tile, the halo layout and the descriptors are those of
// conv3d_umma_kernel: output tiles of tz x 16 x 8 voxels (M = 128 rows, one
// per h-w position of a slice), N = cout, the input halo staged as 16-byte rows
// halo[chunk][position][8 channels] so that every tap is a descriptor offset
// into the same planes.  What changes is who moves the data and when:
//   * warp 0 (one lane) is the producer.  It walks the CTA's tiles and, per
//     tile, the channel groups (cg 8-channel chunks each).  A stage is one
//     (tile, group): one TMA tensor copy per chunk of the NDHWC activation, box
//     (8 ch, 10 w, 18 h, tz + 2 d, 1 n), which the copy engine writes in exactly
//     the plane layout above and fills with zeros outside the tensor (the
//     convolution's padding); where the weights do not fit shared memory for
//     the whole launch, one TMA copy per 8-channel weight chunk (box 8 x cout of
//     the [cout][kpad] matrix) joins the stage.  The innermost coordinate of
//     every copy is a multiple of 8 bf16 = 16 bytes.
//   * warp 1 issues the tcgen05.mma of each stage into one of two
//     accumulators in tensor memory, commits each stage to release its buffer
//     to the producer and each finished tile to the epilogue.
//   * warps 2-5 drain an accumulator (tcgen05.ld, bias, ReLU, bf16 stores, one
//     output voxel per thread) and release it.
// With streamed weights the output channels may be split into parts, each a tile of its
// own (ws_plan).  Resident weights are staged once per block as [group][chunks in the order of
// w_place][cout][8].
// With one channel group and resident weights the MMAs of a slice are issued
// in the order of conv3d_umma_kernel, so the two produce identical bits.
// Every mbarrier wait gives up after kUWaitNs, records the failure in shared
// memory and in g_umma_failures, and every role then leaves its loop; the
// producer waits (bounded) for its copies in flight and the MMA warp for its
// MMAs before the tensor memory is freed.  No multicast anywhere.
#pragma once

#include <cuda.h>

namespace pmd {

constexpr int kWsThreads = 192;  // producer warp, MMA warp, four epilogue warps
constexpr int kWsMaxStages = 4;

struct WsConv {
    ConvShape s;
    int tz;                  // output d-slices per tile
    int tiles_d, tiles_h, tiles_w, n_tiles;
    int cg;                  // 8-channel chunks per stage (channel group)
    int groups;              // stages per tile: cin / 8 / cg
    int stages;              // stage buffers in shared memory
    int streamed;            // 1: weights travel with every stage; 0: resident for the launch
    unsigned plane_bytes;    // stride between halo planes (a box, rounded up to 128 bytes)
    unsigned box_bytes;      // bytes one halo copy writes
    unsigned halo_part;      // cg planes + zeroed slack: offset of a stage's weights
    unsigned stage_bytes;    // stride between stage buffers
    unsigned w_chunks;       // weight chunks of one channel group (cg = 1: with the zero partners)
    unsigned tx_bytes;       // bytes the copy engine writes per stage
    unsigned acc_cols;       // tensor-memory columns of one accumulator: tz * cout
    unsigned tmem_cols;      // allocated: two accumulators, a power of two >= 32
    int ystride;             // channels per voxel of the output tensor
    int parts;               // streamed weights: output-channel parts, each a tile of its own with s.cout = N channels
    int split;               // 8-channel chunks of the first input tensor (cin / 8 where it is the only one)
    // conv3d_zs_kernel: output slices instead of tiles (n_tiles counts them), those of
    // one (h, w) tile after another
    int line;                // slices of a tile, d rounded up to even; 0: tiles
    int share;               // slices of a block, even
    int run;                 // most slices of a run, even; line unless the groups take whole runs
    int ring;                // a power of two: accumulator batches (of kRunSlices) in tensor memory
};

// An optional 1x1x1 head fused into the epilogue: out[m] = b + base[m] +
// sum_c w[c] * y[m][c] over the bf16 outputs, which are then not stored.
struct WsHead {
    const float* w = nullptr;     // [cout]; null: no head, y is written
    const float* b = nullptr;     // [1]
    const float* base = nullptr;  // [voxels] or null
    float* out = nullptr;         // [voxels]
};

__device__ __forceinline__ void mbar_arrive_expect_tx(uint32_t mbar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(mbar), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t mbar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(mbar) : "memory");
}

__device__ __forceinline__ void tma_load_5d(uint32_t dst, const CUtensorMap* map, int c0, int c1,
                                            int c2, int c3, int c4, uint32_t mbar) {
    asm volatile(
        "cp.async.bulk.tensor.5d.shared::cluster.global.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%2, %3, %4, %5, %6}], [%7];" ::"r"(dst),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(c4), "r"(mbar)
        : "memory");
}
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int c0, int c1,
                                            uint32_t mbar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(mbar)
        : "memory");
}

// Bounded wait for the completion of phase `parity`: false once kUWaitNs have
// passed (the shared failure flag is then set) or another role has failed.
__device__ __forceinline__ bool ws_wait(uint32_t mbar, uint32_t parity, volatile int* failed) {
    if (mbar_try(mbar, parity)) return true;
    const unsigned long long start = global_ns();
    while (!mbar_try(mbar, parity)) {
        if (*failed) return false;
        if (global_ns() - start > kUWaitNs) {
            *failed = 1;
            return false;
        }
    }
    return true;
}

// The same for a whole warp, with an answer that is uniform to the compiler.
__device__ __forceinline__ bool ws_wait_warp(uint32_t mbar, uint32_t parity, volatile int* failed) {
    return __all_sync(0xffffffffu, ws_wait(mbar, parity, failed));
}

__device__ __forceinline__ void ws_tile_origin(const WsConv& p, int tile, int& nb, int& z0, int& y0,
                                               int& x0) {
    int t = tile;
    const int tx = t % p.tiles_w;
    t /= p.tiles_w;
    const int ty = t % p.tiles_h;
    t /= p.tiles_h;
    const int tzi = t % p.tiles_d;
    nb = t / p.tiles_d;
    z0 = tzi * p.tz;
    y0 = ty * kUTY;
    x0 = tx * kUTX;
}

// Plane q of a stage: 8-channel chunk `chunk` of the input, whose chunks from p.split on
// are another tensor's (a skip connection that was not copied behind the upsampled one).
__device__ __forceinline__ void ws_load_plane(const WsConv& p, uint32_t dst, const CUtensorMap* x,
                                              const CUtensorMap* skip, int chunk, int q, int cx, int cy, int cz, int cn,
                                              uint32_t mbar) {
    const bool second = chunk >= p.split;
    tma_load_5d(dst + (uint32_t)q * p.plane_bytes, second ? skip : x, (second ? chunk - p.split : chunk) * 8, cx, cy,
                cz, cn, mbar);
}

// The weights of every group into shared memory, [group][w_place][cout][8].  Eight
// 16-byte loads in flight per thread: one at a time, the 10,368 of the 96 -> 32 layer
// took 40 us of each launch.
template <int CG>
__device__ __forceinline__ void ws_stage_weights(unsigned char* wres, const __nv_bfloat16* __restrict__ wt,
                                                 const WsConv& p, int tid) {
    const int N = p.s.cout, cpt = p.s.cin / 8, total = p.groups * (int)p.w_chunks * N;
    for (int i0 = tid; i0 < total; i0 += 8 * kWsThreads) {
        uint4 v[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const int i = i0 + k * kWsThreads, n = i % N, c = i / N;
            const int g = c / (int)p.w_chunks, jj = c % (int)p.w_chunks;
            const int in_group = w_chunk_at(jj, CG);  // tap * CG + q
            const int chunk = in_group / CG * cpt + g * CG + in_group % CG;
            v[k] = make_uint4(0u, 0u, 0u, 0u);  // the CG = 1 zero partner
            if (g < p.groups && in_group < 27 * CG)
                v[k] = __ldg(reinterpret_cast<const uint4*>(wt + (long long)n * p.s.kpad + chunk * 8));
        }
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const int i = i0 + k * kWsThreads;
            if (i < total) *reinterpret_cast<uint4*>(wres + (size_t)i * 16) = v[k];
        }
    }
}

// The epilogue of one accumulator slice (columns from `acc` on), one output voxel per
// thread: bias, ReLU, bf16 stores, or the fused head.  in: whether the thread's voxel
// m lies in the volume; hbase: its value of head.base.
__device__ __forceinline__ void ws_store_slice(const WsConv& p, uint32_t acc, bool in, long long m, int quarter,
                                               const float* bias, __nv_bfloat16* __restrict__ y, int relu,
                                               const WsHead& head, const float* hw, float hbase) {
    const ConvShape& s = p.s;
    __nv_bfloat16* out = y + m * p.ystride;
    // the fused head: bias + base + its weights over the stored bf16
    // channel values, in channel order (pmd_head's arithmetic)
    float hacc = 0.0f;
    if (hw && in) hacc = __ldg(head.b) + hbase;
    for (int c = 0; c < s.cout / 16; ++c) {
        float v[16];
        tmem_ld16(acc + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(c * 16), v);
        if (in) {
            union {
                uint4 u4[2];
                __nv_bfloat162 h[8];
            } pk;
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                float lo = v[2 * e], hi = v[2 * e + 1];
                if (bias) {
                    lo += bias[c * 16 + 2 * e];
                    hi += bias[c * 16 + 2 * e + 1];
                }
                if (relu) {
                    lo = fmaxf(lo, 0.0f);
                    hi = fmaxf(hi, 0.0f);
                }
                pk.h[e] = __floats2bfloat162_rn(lo, hi);
            }
            if (hw) {
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    hacc += hw[c * 16 + 2 * e] * __low2float(pk.h[e]);
                    hacc += hw[c * 16 + 2 * e + 1] * __high2float(pk.h[e]);
                }
            } else {
                uint4* o = reinterpret_cast<uint4*>(out + c * 16);
                o[0] = pk.u4[0];
                o[1] = pk.u4[1];
            }
        }
    }
    if (hw && in) head.out[m] = hacc;
}

// CG = cg, the 8-channel chunks of a stage.
template <int CG>
__global__ void __launch_bounds__(kWsThreads, 1)
conv3d_ws_kernel(const __grid_constant__ CUtensorMap xmap, const __grid_constant__ CUtensorMap skip_map,
                 const __grid_constant__ CUtensorMap wmap,
                 const __nv_bfloat16* __restrict__ wt, const float* __restrict__ bias,
                 __nv_bfloat16* __restrict__ y, WsConv p, int relu, WsHead head) {
    extern __shared__ __align__(1024) unsigned char smem[];
    const ConvShape& s = p.s;
    const int N = s.cout;
    const int cpt = s.cin / 8, S = p.stages;
    constexpr int cg = CG;
    const int tid = threadIdx.x, warp = warp_index(), lane = tid & 31;
    unsigned char* stage0 = smem;  // stage b at stage0 + b * stage_bytes
    unsigned char* wres = smem + (size_t)S * p.stage_bytes;  // resident weights (streamed: empty)
    // resident weights: [group][w_place][cout][8], w_chunks per group
    const size_t group_bytes = (size_t)p.w_chunks * N * 16;
    const size_t wres_bytes = p.streamed ? 0 : (size_t)p.groups * group_bytes;
    uint64_t* bars = reinterpret_cast<uint64_t*>(wres + wres_bytes);  // full[S], empty[S], acc_full[2], acc_free[2]
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * S + 4);
    volatile int* failed = reinterpret_cast<volatile int*>(tmem_slot + 1);
    const uint32_t st_s = smem_u32(stage0), bar_s = smem_u32(bars);
    const uint32_t wbase = p.streamed ? st_s + p.halo_part : smem_u32(wres);
    auto full = [&](int b) { return bar_s + 8u * (uint32_t)b; };
    auto empty = [&](int b) { return bar_s + 8u * (uint32_t)(S + b); };
    auto acc_full = [&](int a) { return bar_s + 8u * (uint32_t)(2 * S + a); };
    auto acc_free = [&](int a) { return bar_s + 8u * (uint32_t)(2 * S + 2 + a); };

    // ---- set-up.  The copy engine writes only the boxes and the weight chunks
    // of a stage; the rest of each stage (plane padding, the slack after the
    // planes, with cg = 1 the zero partner of the last tap's weights) is zeroed
    // here once: the cg = 1 tap pairing reads past the last box and multiplies
    // those bytes by the zero weights, so they must be finite.
    for (int b = 0; b < S; ++b) {
        uint32_t* st = reinterpret_cast<uint32_t*>(stage0 + (size_t)b * p.stage_bytes);
        for (int i = tid; i < (int)(p.halo_part / 4); i += blockDim.x) {
            const unsigned byte = 4u * (unsigned)i;
            if (byte >= (unsigned)cg * p.plane_bytes || byte % p.plane_bytes >= p.box_bytes) st[i] = 0u;
        }
        if (p.streamed && cg == 1)
            for (int i = tid; i < N * 4; i += blockDim.x) st[(p.halo_part + 27u * N * 16u) / 4 + i] = 0u;
    }
    if (!p.streamed) ws_stage_weights<CG>(wres, wt, p, tid);
    if (tid == 0) {
        for (int i = 0; i < 2 * S + 2; ++i) mbar_init(bar_s + 8u * i, 1);
        for (int i = 2 * S + 2; i < 2 * S + 4; ++i) mbar_init(bar_s + 8u * i, 128);
        *failed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_u32(tmem_slot)),
                     "r"(p.tmem_cols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    fence_async_smem();  // zeroed bytes and resident weights are read by the tensor cores
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    if (warp == 0) {
        // ---- producer ----
        if (lane == 0) {
            int st = 0;  // stages issued
            bool stop = false;
            for (int tile = blockIdx.x; tile < p.n_tiles && !stop; tile += gridDim.x) {
                int nb, z0, y0, x0;
                ws_tile_origin(p, tile / p.parts, nb, z0, y0, x0);
                for (int g = 0; g < p.groups; ++g) {
                    const int b = st % S, use = st / S;
                    if (use >= 1 && !ws_wait(empty(b), (uint32_t)((use - 1) & 1), failed)) {
                        stop = true;
                        break;
                    }
                    mbar_arrive_expect_tx(full(b), p.tx_bytes);
                    const uint32_t dst = st_s + (uint32_t)b * p.stage_bytes;
                    for (int q = 0; q < cg; ++q)
                        ws_load_plane(p, dst, &xmap, &skip_map, g * cg + q, q, x0 - 1, y0 - 1, z0 - 1, nb, full(b));
                    if (p.streamed)
                        for (int tap = 0; tap < 27; ++tap)
                            for (int q = 0; q < cg; ++q)
                                tma_load_2d(dst + p.halo_part + (uint32_t)w_place(tap, q, cg) * N * 16, &wmap,
                                            (tap * cpt + g * cg + q) * 8, tile % p.parts * N, full(b));
                    ++st;
                }
            }
            // copies still in flight land before the block can exit
            for (int t = st > S ? st - S : 0; t < st; ++t) mbar_wait(full(t % S), (uint32_t)((t / S) & 1));
        }
    } else if (warp == 1) {
        // ---- MMA issuer: the warp runs the loops, one lane issues ----
        const uint32_t lead = elect_lane();
        int st = 0, last = -1;  // stages consumed; the last one committed
        bool stop = false;
        for (int i = 0, tile = blockIdx.x; tile < p.n_tiles && !stop; ++i, tile += gridDim.x) {
            const int a = i & 1;
            if (i >= 2 && !ws_wait_warp(acc_free(a), (uint32_t)(((i >> 1) & 1) ^ 1), failed)) break;
            tc_fence_after();
            const uint32_t d0 = tmem + (uint32_t)a * p.acc_cols;
            for (int g = 0; g < p.groups; ++g, ++st) {
                const int b = st % S;
                if (!ws_wait_warp(full(b), (uint32_t)((st / S) & 1), failed)) {
                    stop = true;
                    break;
                }
                tc_fence_after();
                const uint32_t stage = st_s + (uint32_t)b * p.stage_bytes;
                const uint32_t wg = p.streamed ? stage + p.halo_part
                                               : wbase + (uint32_t)((size_t)g * group_bytes);
                umma_issue_taps<CG>(d0, stage, p.plane_bytes, wg, N, p.tz, g > 0, lead);
                umma_commit(empty(b), lead);
                last = st;
            }
            if (!stop) umma_commit(acc_full(a), lead);
        }
        // MMAs still in flight finish before the tensor memory is freed
        if (last >= 0) mbar_wait(empty(last % S), (uint32_t)((last / S) & 1));
    } else {
        // ---- epilogue: one accumulator row (output voxel) per thread ----
        const int quarter = warp & 3;  // the tensor-memory lanes this warp may read
        const int r = quarter * 32 + lane;
        for (int i = 0, tile = blockIdx.x; tile < p.n_tiles; ++i, tile += gridDim.x) {
            const int a = i & 1;
            int ok = lane == 0 ? (ws_wait(acc_full(a), (uint32_t)((i >> 1) & 1), failed) ? 1 : 0) : 0;
            ok = __shfl_sync(0xffffffffu, ok, 0);  // the warp leaves or reads together
            if (!ok) break;
            tc_fence_after();
            int nb, z0, y0, x0;
            ws_tile_origin(p, tile / p.parts, nb, z0, y0, x0);
            const int yg = y0 + r / kUTX, xg = x0 + r % kUTX, n0 = tile % p.parts * N;  // the part's first channel
            for (int sl = 0; sl < p.tz; ++sl) {
                const int z = z0 + sl;
                const bool in = z < s.d && yg < s.h && xg < s.w;
                const long long m =
                    (((long long)nb * s.d + (in ? z : 0)) * s.h + (in ? yg : 0)) * s.w + (in ? xg : 0);
                ws_store_slice(p, tmem + (uint32_t)a * p.acc_cols + (uint32_t)(sl * N), in, m, quarter,
                               bias ? bias + n0 : nullptr, y + n0, relu, head, head.w,
                               in && head.w && head.base ? head.base[m] : 0.0f);
            }
            tc_fence_before();
            mbar_arrive(acc_free(a));
        }
    }

    tc_fence_before();
    __syncthreads();
    if (tid == 0 && *failed) atomicAdd(&g_umma_failures, 1);
    if (warp == 0) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                     "r"(p.tmem_cols)
                     : "memory");
    }
}

// ---- runs along d --------------------------------------------------------------------
// Where the weights are resident and three outputs fit one MMA (3 cout <= 256), a block
// walks along d instead of taking tiles: a stage holds T = 2 halo slices without the d
// halo (every slice of a run is fetched once; tiles of two slices fetched each
// twice, and the copy engine, which moves these 16-byte rows, was as busy as the
// tensor cores), and halo slice i always adds to outputs i - 2, i - 1 and i of the run:
// N = 3 cout for all but the run's first and last slices.  Chunk c, halo slices
// [c T, c T + T), completes the batch of outputs [c T - 2, c T + T - 2).  Channel group
// g follows two chunks behind group g - 1: an output has all its slices of one group
// before the first of the next, the order of the tiles.  Where the ring cannot hold so
// many batches (96 -> 32 has six groups) a group takes the whole run before the next
// one starts, and a run is as long as the ring.  The
// accumulators of `ring` batches lie one after another in tensor memory, used in
// turn across runs; an MMA that reaches past the last one is split there.  A block takes
// an equal share of all slices, whatever tile they lie in.  With its operands uniform
// (umma_bf16) and no division in its loop the issuing warp is no longer the bound: what
// is left is shared memory, which the MMAs read and the copies write 16 bytes a row
// (two cycles a row, 360 rows a slice at 16 channels).  Roles,
// waits, failure handling and the order of an output's products as above.
constexpr int kRunSlices = 2;  // halo slices of a stage, output slices of a batch

template <int CG>
__global__ void __launch_bounds__(kWsThreads, 1)
conv3d_zs_kernel(const __grid_constant__ CUtensorMap xmap, const __grid_constant__ CUtensorMap skip_map,
                 const __nv_bfloat16* __restrict__ wt,
                 const float* __restrict__ bias, __nv_bfloat16* __restrict__ y, WsConv p, int relu, WsHead head) {
    extern __shared__ __align__(1024) unsigned char smem[];
    const ConvShape& s = p.s;
    const int N = s.cout, S = p.stages, T = kRunSlices, RB = p.ring;
    const int tid = threadIdx.x, warp = warp_index(), lane = tid & 31;
    unsigned char* wres = smem + (size_t)S * p.stage_bytes;
    const size_t group_bytes = (size_t)p.w_chunks * N * 16;
    // full[S], empty[S], acc_full[RB], acc_free[RB]
    uint64_t* bars = reinterpret_cast<uint64_t*>(wres + (size_t)p.groups * group_bytes);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * S + 2 * RB);
    volatile int* failed = reinterpret_cast<volatile int*>(tmem_slot + 1);
    // the epilogue's bias and head weights (16 bytes after the barriers)
    float* sbias = reinterpret_cast<float*>(bars + 2 * S + 2 * RB + 2);
    float* shead = sbias + N;
    const uint32_t st_s = smem_u32(smem), bar_s = smem_u32(bars), w_s = smem_u32(wres);
    auto full = [&](int b) { return bar_s + 8u * (uint32_t)b; };
    auto empty = [&](int b) { return bar_s + 8u * (uint32_t)(S + b); };
    auto acc_full = [&](int a) { return bar_s + 8u * (uint32_t)(2 * S + a); };
    auto acc_free = [&](int a) { return bar_s + 8u * (uint32_t)(2 * S + RB + a); };

    ws_stage_weights<CG>(wres, wt, p, tid);
    for (int i = tid; i < N; i += kWsThreads) {
        sbias[i] = bias ? bias[i] : 0.0f;
        if (head.w) shead[i] = head.w[i];
    }
    if (tid == 0) {
        for (int i = 0; i < 2 * S + RB; ++i) mbar_init(bar_s + 8u * i, 1);
        for (int i = 2 * S + RB; i < 2 * S + 2 * RB; ++i) mbar_init(bar_s + 8u * i, 128);
        *failed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_u32(tmem_slot)),
                     "r"(p.tmem_cols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    fence_async_smem();  // the weights are read by the tensor cores
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    // this block's slices, and the run that begins at `at`: batch item, first output
    // slice, slices, tile corner; returns where the next one begins
    const int at0 = (int)blockIdx.x * p.share, at1 = min(at0 + p.share, p.n_tiles);
    auto run_at = [&](int at, int& nb, int& z0, int& len, int& y0, int& x0) {
        int t = at / p.line;
        z0 = at % p.line;
        const int next = min(min(at1, at - z0 + p.line), at + p.run);
        len = min(next - at, s.d - z0);
        x0 = t % p.tiles_w * kUTX;
        t /= p.tiles_w;
        y0 = t % p.tiles_h * kUTY;
        nb = t / p.tiles_h;
        return next;
    };
    auto chunks_of = [&](int len) { return (len + 2 + T - 1) / T; };
    // chunks by which a channel group follows the one before
    auto lag_of = [&](int n_chunks) { return p.run < p.line ? n_chunks : 2; };

    if (warp == 0) {
        // ---- producer ----
        if (lane == 0) {
            int st = 0, b = 0;         // stages issued, the next one's buffer
            uint32_t free_phase = 1u;  // the buffers' first use waits for nothing
            bool stop = false;
            for (int at = at0; at < at1 && !stop;) {
                int nb, z0, len, y0, x0;
                at = run_at(at, nb, z0, len, y0, x0);
                const int n_chunks = chunks_of(len), lag = lag_of(n_chunks);
                for (int step = 0; step < n_chunks + lag * (p.groups - 1) && !stop; ++step)
                    for (int g = 0; g < p.groups; ++g) {
                        const int c = step - lag * g;
                        if (c < 0 || c >= n_chunks) continue;
                        if (!ws_wait(empty(b), free_phase, failed)) {
                            stop = true;
                            break;
                        }
                        mbar_arrive_expect_tx(full(b), p.tx_bytes);
                        const uint32_t dst = st_s + (uint32_t)b * p.stage_bytes;
                        for (int q = 0; q < CG; ++q)
                            ws_load_plane(p, dst, &xmap, &skip_map, g * CG + q, q, x0 - 1, y0 - 1, z0 - 1 + c * T, nb,
                                          full(b));
                        ++st;
                        if (++b == S) {
                            b = 0;
                            free_phase ^= 1u;
                        }
                    }
            }
            // copies still in flight land before the block can exit
            for (int t = st > S ? st - S : 0; t < st; ++t) mbar_wait(full(t % S), (uint32_t)((t / S) & 1));
        }
    } else if (warp == 1) {
        // ---- MMA issuer: the warp runs the loops, one lane issues ----
        const uint32_t lead = elect_lane();
        constexpr uint64_t slice16 = (uint64_t)(kUHY * kUHX);
        const uint64_t plane16 = p.plane_bytes >> 4;
        const int R = RB * T;
        int b = 0, last = -1;                // the next stage's buffer; the last one committed
        uint32_t phase = 0u, last_phase = 0u;
        int batch = 0;                       // batches of the runs before
        int next = 0;                        // and of the next one to acquire
        uint32_t next_phase = 1u;            // the first round through the ring waits for nothing
        bool stop = false;
        for (int at = at0; at < at1 && !stop;) {
            int nb, z0, len, y0, x0;
            at = run_at(at, nb, z0, len, y0, x0);
            const int n_chunks = chunks_of(len), lag = lag_of(n_chunks);
            int owned = 0;  // batches of this run free to write
            for (int step = 0; step < n_chunks + lag * (p.groups - 1) && !stop; ++step) {
                // the batch that group 0 goes on with and the one it begins
                for (; owned < min(step + 2, n_chunks) && !stop; ++owned) {
                    stop = !ws_wait_warp(acc_free(next), next_phase, failed);
                    if (++next == RB) {
                        next = 0;
                        next_phase ^= 1u;
                    }
                }
                if (stop) break;
                tc_fence_after();
                for (int g = 0; g < p.groups; ++g) {
                    const int c = step - lag * g;
                    if (c < 0 || c >= n_chunks) continue;
                    if (!ws_wait_warp(full(b), phase, failed)) {
                        stop = true;
                        break;
                    }
                    tc_fence_after();
                    const int place = (batch + c) & (RB - 1);  // of batch c
                    const uint64_t a0 = umma_smem_desc(st_s + (uint32_t)b * p.stage_bytes, p.plane_bytes, kUHX * 16);
                    const uint64_t b0 =
                        umma_smem_desc(w_s + (uint32_t)((size_t)g * group_bytes), 3u * (uint32_t)N * 16, 128);
#pragma unroll 1
                    for (int k = 0; k < T; ++k) {
                        const int i = c * T + k;  // halo slice of the run: z0 - 1 + i
                        const int hi = min(i, len - 1);
#pragma unroll 1
                        for (int lo = max(i - 2, 0); lo <= hi;) {
                            int slot = place * T + lo + 2 - c * T;  // output lo's ring slot
                            if (slot >= R) slot -= R;
                            const int cnt = min(hi - lo + 1, R - slot);
                            umma_issue_slice<CG>(tmem + (uint32_t)(slot * N), a0 + slice16 * (uint64_t)k,
                                                 b0 + (uint64_t)((2 - i + lo) * N), plane16, N, cnt,
                                                 g == 0 && lo + cnt - 1 == i, lead);
                            lo += cnt;
                        }
                    }
                    umma_commit(empty(b), lead);
                    last = b;
                    last_phase = phase;
                    if (++b == S) {
                        b = 0;
                        phase ^= 1u;
                    }
                    if (g == p.groups - 1) umma_commit(acc_full(place), lead);
                }
            }
            batch += n_chunks;
        }
        // MMAs still in flight finish before the tensor memory is freed
        if (last >= 0) mbar_wait(empty(last), last_phase);
    } else {
        // ---- epilogue: one accumulator row (output voxel) per thread ----
        const int quarter = warp & 3;  // the tensor-memory lanes this warp may read
        const int r = quarter * 32 + lane;
        int a = 0;  // ring place of the batch
        uint32_t phase = 0u;
        bool stop = false;
        for (int at = at0; at < at1 && !stop;) {
            int nb, z0, len, y0, x0;
            at = run_at(at, nb, z0, len, y0, x0);
            const int yg = y0 + r / kUTX, xg = x0 + r % kUTX;
            const bool in = yg < s.h && xg < s.w;
            const long long m0 = (((long long)nb * s.d + z0) * s.h + (in ? yg : 0)) * s.w + (in ? xg : 0);
            for (int c = 0; c < chunks_of(len); ++c) {
                // the head's base values are fetched while the accumulators are waited for
                float hbase[kRunSlices] = {};
                if (head.base && in)
#pragma unroll
                    for (int k = 0; k < kRunSlices; ++k) {
                        const int o = c * kRunSlices + k - 2;
                        if (o >= 0 && o < len) hbase[k] = __ldg(head.base + m0 + (long long)o * s.h * s.w);
                    }
                int ok = lane == 0 ? (ws_wait(acc_full(a), phase, failed) ? 1 : 0) : 0;
                ok = __shfl_sync(0xffffffffu, ok, 0);  // the warp leaves or reads together
                if (!ok) {
                    stop = true;
                    break;
                }
                tc_fence_after();
#pragma unroll
                for (int k = 0; k < kRunSlices; ++k) {
                    const int o = c * kRunSlices + k - 2;
                    if (o >= 0 && o < len)
                        ws_store_slice(p, tmem + (uint32_t)((a * kRunSlices + k) * N), in,
                                       m0 + (long long)o * s.h * s.w, quarter, bias ? sbias : nullptr, y, relu, head,
                                       head.w ? shead : nullptr, hbase[k]);
                }
                tc_fence_before();
                mbar_arrive(acc_free(a));
                if (++a == RB) {
                    a = 0;
                    phase ^= 1u;
                }
            }
        }
    }

    tc_fence_before();
    __syncthreads();
    if (tid == 0 && *failed) atomicAdd(&g_umma_failures, 1);
    if (warp == 0) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                     "r"(p.tmem_cols)
                     : "memory");
    }
}

}  // namespace pmd
