// pmc_presolve.cu — the treatment-head pre-solve on the GPU (C-ABI in
// include/pyradmc_b200_presolve.h).
//
// One thread per primary traces it through the beam-limiting stack and the
// air column (geometry/head.py:373-575 is the algorithm; the chord lengths
// restate the scalar twins of geometry/collimation.py:253-490) and writes its
// exit-plane particles into fixed slots (transmitted, stack scatter, air
// photon, air electron), so the output order is the primaries' order whatever
// the scheduling; a block count, a prefix sum and a block-local rank then
// compact the kept slots.  Random numbers: the Philox stream of (seed,
// primary index) under a tag of its own.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <vector>

#include "../../include/pyradmc_b200.h"
#include "../../include/pyradmc_b200_presolve.h"
#include "pmc_common.cuh"
#include "pmc_physics.cuh"
#include "pmc_scan.cuh"
#include "pmc_stack.cuh"

namespace pmc_head {

using pmc::Rng;

constexpr int kThreads = 256;
constexpr uint32_t kHeadTag = 0x48454144u;  // stream tag of the pre-solve ("HEAD")

struct Params {
    int first_compton, has_air, air_row;
    float air_z0, air_z1, exit_z, pcut, ecut, floor;
    uint32_t seed_lo, seed_hi;
};

// The primaries: coordinate k of primary i at pos[i * primary + k * axis] (records
// of three: 3 and 1; columns: 1 and n), dir alike.
struct In {
    const float* energy;
    const float* pos;
    const float* dir;
    const float* weight;
    long long primary, axis;
};

// One exit-plane slot; kind 0 = empty.
struct Out {
    int* kind;
    float* energy;
    float* pos;
    float* dir;
    float* weight;
};

// head.py:319-337: a secondary below the floor survives with probability
// w / floor at weight floor.
__device__ __forceinline__ float roulette(float w, float floor, Rng& rng) {
    if (floor <= 0.0f || w <= 0.0f || w >= floor) return w;
    return rng.uniform() < w / floor ? floor : 0.0f;
}

// A kept particle slides straight to the exit plane into its slot; a dropped
// one adds its weight x energy to `dropped` (head.py:576-599).
__device__ __forceinline__ void emit(const Stack& S, const Params& P, const Out& o, long long slot, int kind,
                                     float e, const float* x, const float* u, float w, float cutoff,
                                     double& dropped) {
    bool kept = false;
    if (w > 0.0f && e >= cutoff) {
        const float d_w = S.rot[6] * u[0] + S.rot[7] * u[1] + S.rot[8] * u[2];
        if (d_w > 0.0f) {
            const float p_w = S.rot[6] * (x[0] - S.origin[0]) + S.rot[7] * (x[1] - S.origin[1]) +
                              S.rot[8] * (x[2] - S.origin[2]);
            const float t = (P.exit_z - p_w) / d_w;
            if (t >= 0.0f) {
                kept = true;
                o.kind[slot] = kind;
                o.energy[slot] = e;
                o.weight[slot] = w;
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    o.pos[3 * slot + k] = x[k] + t * u[k];
                    o.dir[3 * slot + k] = u[k];
                }
            }
        }
    }
    if (!kept) dropped += (double)w * (double)e;
}

__global__ void __launch_bounds__(kThreads) presolve_kernel(Stack S, Mu M, Params P, long long n, In in, Out o,
                                                          int per_primary, double* __restrict__ block_dropped) {
    __shared__ double red[kThreads / 32];
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    double dropped = 0.0;
    if (i < n) {
        const float e = in.energy[i], w = in.weight[i];
        const float* pos = in.pos + i * in.primary;
        const float* dir = in.dir + i * in.primary;
        const float x[3] = {pos[0], pos[in.axis], pos[2 * in.axis]};
        const float u[3] = {dir[0], dir[in.axis], dir[2 * in.axis]};
        float pl[3], dl[3];
        to_local(S, x, u, pl, dl);
        Rng rng;
        rng.load(P.seed_lo, P.seed_hi, pmc::StreamId{(uint32_t)i, (uint32_t)(i >> 32), kHeadTag, 0u});
        long long slot = i * per_primary;
        const long long s_trans = slot++;

        // ---- the stack (head.py:424-484) ----
        float tau[kMaxDevices];
        float tau_total = 0.0f;
        for (int j = 0; j < S.n; ++j) {
            tau[j] = mu_at(M, M.log_total, j, e) * device_len(S, j, pl, dl, 0);
            tau_total += tau[j];
        }
        float trans_w = w * expf(-tau_total);
        if (P.first_compton) {
            const long long s_scat = slot++;
            if (tau_total > 0.0f) {
                // the device by its share of the optical depth; the site at its
                // mid-plane crossing (the stated approximation of head.py:37-41)
                const float pick = rng.uniform() * tau_total;
                int jd = S.n - 1;
                float acc = 0.0f;
                for (int j = 0; j < S.n; ++j) {
                    acc += tau[j];
                    if (pick <= acc) {
                        jd = j;
                        break;
                    }
                }
                const float z_mid = 0.5f * (S.z_top[jd] + S.z_bottom[jd]);
                const float t_mid = (z_mid - pl[2]) / dl[2];
                const float site[3] = {x[0] + t_mid * u[0], x[1] + t_mid * u[1], x[2] + t_mid * u[2]};
                const float cf = mu_at(M, M.log_compton, jd, e) / mu_at(M, M.log_total, jd, e);
                const float iw = w * (1.0f - expf(-tau_total));
                const float ratio = pmc::sample_compton_energy_ratio(e, rng);
                const float e_out = ratio * e;
                const float phi = pmc::kTwoPi * rng.uniform();
                float d_out[3] = {u[0], u[1], u[2]};
                pmc::rotate_direction(d_out[0], d_out[1], d_out[2], pmc::compton_cos_theta(e, ratio), phi);
                float sl[3], sd[3];
                to_local(S, site, d_out, sl, sd);
                float tau_out = 0.0f;
                for (int j = 0; j < S.n; ++j)
                    tau_out += mu_at(M, M.log_total, j, e_out) * device_len(S, j, sl, sd, 1);
                const float sw = roulette(iw * cf * expf(-tau_out), P.floor, rng);
                emit(S, P, o, s_scat, 1, e_out, site, d_out, sw, P.pcut, dropped);
            }
        }

        // ---- the air column, primaries only (head.py:487-553) ----
        if (P.has_air) {
            const bool forward = dl[2] > 0.0f;
            const float length = forward ? (P.air_z1 - P.air_z0) / dl[2] : 0.0f;
            const float mu_air = mu_at(M, M.log_total, P.air_row, e);
            const float tau_air = mu_air * length;
            const float pre = trans_w;
            trans_w *= expf(-tau_air);
            if (P.first_compton) {
                const long long s_ph = slot++, s_el = slot++;
                if (forward && tau_air > 0.0f) {
                    const float iw = pre * (1.0f - expf(-tau_air));
                    const float pw = iw * (mu_at(M, M.log_compton, P.air_row, e) / mu_air);
                    const float ud = rng.uniform();
                    const float depth = -logf(1.0f - ud * (1.0f - expf(-tau_air))) / mu_air;
                    const float t0 = (P.air_z0 - pl[2]) / dl[2] + depth;
                    const float site[3] = {x[0] + t0 * u[0], x[1] + t0 * u[1], x[2] + t0 * u[2]};
                    const float ratio = pmc::sample_compton_energy_ratio(e, rng);
                    const float e_ph = ratio * e, e_el = e - e_ph;
                    const float phi = pmc::kTwoPi * rng.uniform();
                    float d_ph[3] = {u[0], u[1], u[2]}, d_el[3] = {u[0], u[1], u[2]};
                    pmc::rotate_direction(d_ph[0], d_ph[1], d_ph[2], pmc::compton_cos_theta(e, ratio), phi);
                    pmc::rotate_direction(d_el[0], d_el[1], d_el[2], pmc::compton_electron_cos_theta(e, ratio),
                                          phi + pmc::kPi);
                    // the two arms are rouletted independently (head.py:528-531)
                    const float w_ph = roulette(pw, P.floor, rng);
                    const float w_el = roulette(pw, P.floor, rng);
                    emit(S, P, o, s_ph, 1, e_ph, site, d_ph, w_ph, P.pcut, dropped);
                    emit(S, P, o, s_el, 2, e_el, site, d_el, w_el, P.ecut, dropped);
                }
            }
        }
        emit(S, P, o, s_trans, 1, e, x, u, trans_w, P.pcut, dropped);
    }
    // per-block dropped weight-energy (summed on the host in block order)
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) dropped += __shfl_xor_sync(0xffffffffu, dropped, off);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = dropped;
    __syncthreads();
    if (threadIdx.x == 0) {
        double s = 0.0;
        for (int k = 0; k < kThreads / 32; ++k) s += red[k];
        block_dropped[blockIdx.x] = s;
    }
}

// Kept slots per block of kThreads consecutive slots.
__global__ void __launch_bounds__(kThreads) count_slots(const int* __restrict__ kind, long long n_slots,
                                                       unsigned int* __restrict__ block_counts) {
    const long long s = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const int keep = s < n_slots && kind[s] != 0;
    const int c = __syncthreads_count(keep);
    if (threadIdx.x == 0) block_counts[blockIdx.x] = (unsigned int)c;
}

// Kept slot s goes to block_offsets[block] + its rank in the block.  kNormalize: as
// the phase space is handed on, directions renormalized and weights scaled by
// particles / n_primaries (head.py:296-314), in float64 and rounded once.
template <bool kNormalize>
__global__ void __launch_bounds__(kThreads) compact_slots(Out in, long long n_slots,
                                                         const unsigned long long* __restrict__ block_offsets,
                                                         const unsigned long long* __restrict__ total,
                                                         long long n_primaries, Out out) {
    __shared__ int warp_base[kThreads / 32];
    const long long s = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const int keep = s < n_slots && in.kind[s] != 0;
    const unsigned int ballot = __ballot_sync(0xffffffffu, keep);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) warp_base[warp] = __popc(ballot);
    __syncthreads();
    if (threadIdx.x == 0) {
        int acc = 0;
        for (int k = 0; k < kThreads / 32; ++k) {
            const int c = warp_base[k];
            warp_base[k] = acc;
            acc += c;
        }
    }
    __syncthreads();
    if (keep) {
        const long long dst =
            (long long)block_offsets[blockIdx.x] + warp_base[warp] + __popc(ballot & ((1u << lane) - 1u));
        out.kind[dst] = in.kind[s];
        out.energy[dst] = in.energy[s];
        float w = in.weight[s], d[3] = {in.dir[3 * s], in.dir[3 * s + 1], in.dir[3 * s + 2]};
        if constexpr (kNormalize) {
            w = (float)__dmul_rn((double)w, __ddiv_rn((double)*total, (double)n_primaries));
            const double x = d[0], y = d[1], z = d[2];
            const double norm = __dsqrt_rn(__dadd_rn(__dadd_rn(__dmul_rn(x, x), __dmul_rn(y, y)), __dmul_rn(z, z)));
            d[0] = (float)__ddiv_rn(x, norm);
            d[1] = (float)__ddiv_rn(y, norm);
            d[2] = (float)__ddiv_rn(z, norm);
        }
        out.weight[dst] = w;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            out.pos[3 * dst + k] = in.pos[3 * s + k];
            out.dir[3 * dst + k] = d[k];
        }
    }
}

__global__ void __launch_bounds__(kThreads) path_lengths_kernel(Stack S, long long n, const float* __restrict__ pos,
                                                               const float* __restrict__ dir, int from_origin,
                                                               float* __restrict__ out) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float pl[3], dl[3];
    to_local(S, pos + 3 * i, dir + 3 * i, pl, dl);
    for (int j = 0; j < S.n; ++j) out[i * S.n + j] = device_len(S, j, pl, dl, from_origin);
}

}  // namespace pmc_head

// ---- host side -------------------------------------------------------------------
namespace {

using namespace pmc_head;

// Device buffers of one call, freed on every exit path.
struct Arena {
    std::vector<void*> ptrs;
    ~Arena() {
        for (void* p : ptrs) cudaFree(p);
    }
    template <typename T>
    T* alloc(size_t n) {
        void* p = nullptr;
        if (cudaMalloc(&p, sizeof(T) * (n > 0 ? n : 1)) != cudaSuccess) return nullptr;
        ptrs.push_back(p);
        return static_cast<T*>(p);
    }
    template <typename T>
    T* upload(const T* src, size_t n) {
        T* d = alloc<T>(n);
        if (d && n && cudaMemcpy(d, src, sizeof(T) * n, cudaMemcpyHostToDevice) != cudaSuccess) return nullptr;
        return d;
    }
    float* upload_f32(const double* src, size_t n) {  // float64 host array -> float32 device array
        std::vector<float> f(n);
        for (size_t i = 0; i < n; ++i) f[i] = (float)src[i];
        return upload(f.data(), n);
    }
};

bool stack_ok(const pmc_head_stack* s) {
    if (!s || s->n_devices < 1 || s->n_devices > kMaxDevices || !s->kind || !s->z_top || !s->z_bottom ||
        !s->jaw_axis || !s->jaw_edge_neg || !s->jaw_edge_pos || !s->jaw_focused || !s->mlc_tip_radius ||
        !s->mlc_focused_sides || !s->mlc_n_pairs || !s->mlc_edges_off || !s->mlc_tips_off)
        return false;
    for (int j = 0; j < s->n_devices; ++j) {
        if (s->kind[j] != 0 && s->kind[j] != 1) return false;
        if (!(s->z_bottom[j] > s->z_top[j])) return false;
        if (s->kind[j] == 0 && s->jaw_axis[j] != 0 && s->jaw_axis[j] != 1) return false;
        if (s->kind[j] == 1) {
            const long long n = s->mlc_n_pairs[j];
            if (n < 0 || s->mlc_edges_off[j] < 0 || s->mlc_tips_off[j] < 0 ||
                s->mlc_edges_off[j] + n + (n > 0 ? 1 : 0) > s->n_leaf_edges ||
                s->mlc_tips_off[j] + n > s->n_tips)
                return false;
            if (n > 0 && (!s->leaf_edges_v || !s->tips_neg || !s->tips_pos)) return false;
        }
    }
    return true;
}

int upload_stack(Arena& a, const pmc_head_stack* s, Stack& S) {
    S.n = s->n_devices;
    for (int k = 0; k < 3; ++k) S.origin[k] = (float)s->origin[k];
    for (int k = 0; k < 9; ++k) S.rot[k] = (float)s->rotation[k];
    const size_t n = (size_t)s->n_devices;
    S.kind = a.upload(s->kind, n);
    S.z_top = a.upload_f32(s->z_top, n);
    S.z_bottom = a.upload_f32(s->z_bottom, n);
    S.jaw_axis = a.upload(s->jaw_axis, n);
    S.jaw_neg = a.upload_f32(s->jaw_edge_neg, n);
    S.jaw_pos = a.upload_f32(s->jaw_edge_pos, n);
    S.jaw_focused = a.upload(s->jaw_focused, n);
    S.tip_radius = a.upload_f32(s->mlc_tip_radius, n);
    S.focused_sides = a.upload(s->mlc_focused_sides, n);
    S.n_pairs = a.upload(s->mlc_n_pairs, n);
    S.edges_off = a.upload(s->mlc_edges_off, n);
    S.tips_off = a.upload(s->mlc_tips_off, n);
    const size_t ne = (size_t)(s->n_leaf_edges > 0 ? s->n_leaf_edges : 0);
    const size_t nt = (size_t)(s->n_tips > 0 ? s->n_tips : 0);
    S.leaf_edges = ne ? a.upload_f32(s->leaf_edges_v, ne) : a.alloc<float>(1);
    S.tips_neg = nt ? a.upload_f32(s->tips_neg, nt) : a.alloc<float>(1);
    S.tips_pos = nt ? a.upload_f32(s->tips_pos, nt) : a.alloc<float>(1);
    const bool ok = S.kind && S.z_top && S.z_bottom && S.jaw_axis && S.jaw_neg && S.jaw_pos && S.jaw_focused &&
                    S.tip_radius && S.focused_sides && S.n_pairs && S.edges_off && S.tips_off && S.leaf_edges &&
                    S.tips_neg && S.tips_pos;
    return ok ? PMC_OK : PMC_ERR_CUDA;
}

int blocks_for(long long n) { return (int)((n + kThreads - 1) / kThreads); }

}  // namespace

extern "C" int pmc_head_path_lengths(const pmc_head_stack* stack, int64_t n, const float* pos, const float* dir,
                                     int32_t from_origin, float* out) {
    if (!stack_ok(stack) || n < 0 || (n > 0 && (!pos || !dir || !out))) return PMC_ERR_INVALID;
    if (n == 0) return PMC_OK;
    Arena a;
    Stack S{};
    if (upload_stack(a, stack, S) != PMC_OK) return PMC_ERR_CUDA;
    const float* dp = a.upload(pos, (size_t)n * 3);
    const float* dd = a.upload(dir, (size_t)n * 3);
    float* dout = a.alloc<float>((size_t)n * stack->n_devices);
    if (!dp || !dd || !dout) return PMC_ERR_CUDA;
    path_lengths_kernel<<<blocks_for(n), kThreads>>>(S, n, dp, dd, from_origin ? 1 : 0, dout);
    if (cudaGetLastError() != cudaSuccess || cudaDeviceSynchronize() != cudaSuccess) return PMC_ERR_CUDA;
    if (cudaMemcpy(out, dout, sizeof(float) * (size_t)n * stack->n_devices, cudaMemcpyDeviceToHost) != cudaSuccess)
        return PMC_ERR_CUDA;
    return PMC_OK;
}

namespace {

// The small arrays of a call, packed for one copy: add() gives an array's offset.
struct Pack {
    std::vector<char> bytes;
    size_t add(const void* src, size_t n) {
        const size_t at = bytes.size();
        bytes.resize(at + (std::max<size_t>(n, 1) + 15) / 16 * 16);
        if (n) std::memcpy(bytes.data() + at, src, n);
        return at;
    }
    size_t ints(const int32_t* src, size_t n) { return add(src, sizeof(int32_t) * n); }
    size_t floats(const double* src, size_t n) {  // float64 host array -> float32
        std::vector<float> f(n);
        for (size_t i = 0; i < n; ++i) f[i] = (float)src[i];
        return add(f.data(), sizeof(float) * n);
    }
};

// One call's plan: checked arguments, the packed tables, and where everything lies
// in the caller's workspace.
struct Plan {
    Pack pack;
    Stack S{};
    Mu M{};
    Params P{};
    long long n = 0, n_slots = 0;
    int per_primary = 1, blocks = 0, slot_blocks = 0;
    size_t tables = 0, columns = 0, kind = 0, energy = 0, pos = 0, dir = 0, weight = 0, drop = 0, counts = 0,
           offsets = 0, totals = 0, packed = 0, bytes = 0;
    size_t at[16];  // offsets into the packed tables
};

int make_plan(const pmc_head_stack* stack, const pmc_head_mu* mu, const pmc_head_params* params, int64_t n,
              bool host_outputs, Plan& p) {
    if (!stack_ok(stack) || !mu || !params || n < 1) return PMC_ERR_INVALID;
    const int rows = stack->n_devices + (params->has_air ? 1 : 0);
    if (mu->n_table < 2 || mu->n_rows < rows || !mu->log_energy || !mu->log_total || !mu->log_compton)
        return PMC_ERR_INVALID;
    if (params->has_air && (params->air_row < 0 || params->air_row >= mu->n_rows)) return PMC_ERR_INVALID;
    const double span = mu->log_energy[mu->n_table - 1] - mu->log_energy[0];
    if (!(span > 0.0)) return PMC_ERR_INVALID;
    const int fc = params->first_compton ? 1 : 0, air = params->has_air ? 1 : 0;
    p.per_primary = 1 + fc * (1 + 2 * air);
    p.n = n;
    p.n_slots = (long long)n * p.per_primary;
    p.blocks = blocks_for(p.n);
    p.slot_blocks = blocks_for(p.n_slots);

    const size_t nd = (size_t)stack->n_devices;
    p.S.n = stack->n_devices;
    for (int k = 0; k < 3; ++k) p.S.origin[k] = (float)stack->origin[k];
    for (int k = 0; k < 9; ++k) p.S.rot[k] = (float)stack->rotation[k];
    const size_t ne = (size_t)(stack->n_leaf_edges > 0 ? stack->n_leaf_edges : 0);
    const size_t nt = (size_t)(stack->n_tips > 0 ? stack->n_tips : 0);
    const size_t n_mu = (size_t)mu->n_rows * mu->n_table;
    size_t* at = p.at;
    *at++ = p.pack.ints(stack->kind, nd);
    *at++ = p.pack.floats(stack->z_top, nd);
    *at++ = p.pack.floats(stack->z_bottom, nd);
    *at++ = p.pack.ints(stack->jaw_axis, nd);
    *at++ = p.pack.floats(stack->jaw_edge_neg, nd);
    *at++ = p.pack.floats(stack->jaw_edge_pos, nd);
    *at++ = p.pack.ints(stack->jaw_focused, nd);
    *at++ = p.pack.floats(stack->mlc_tip_radius, nd);
    *at++ = p.pack.ints(stack->mlc_focused_sides, nd);
    *at++ = p.pack.ints(stack->mlc_n_pairs, nd);
    *at++ = p.pack.ints(stack->mlc_edges_off, nd);
    *at++ = p.pack.ints(stack->mlc_tips_off, nd);
    *at++ = p.pack.floats(stack->leaf_edges_v, ne);
    *at++ = p.pack.floats(stack->tips_neg, nt);
    *at++ = p.pack.floats(stack->tips_pos, nt);
    *at = p.pack.floats(mu->log_total, n_mu);
    p.pack.floats(mu->log_compton, n_mu);  // right behind log_total's block
    p.M.n_rows = mu->n_rows;
    p.M.n_table = mu->n_table;
    p.M.log_e0 = (float)mu->log_energy[0];
    p.M.inv_dlog = (float)((mu->n_table - 1) / span);
    p.P.first_compton = fc;
    p.P.has_air = air;
    p.P.air_row = params->air_row;
    p.P.air_z0 = (float)params->air_z_start;
    p.P.air_z1 = (float)params->air_z_end;
    p.P.exit_z = (float)params->exit_z;
    p.P.pcut = (float)params->pcut;
    p.P.ecut = (float)params->ecut;
    p.P.floor = (float)params->weight_floor;
    p.P.seed_lo = (uint32_t)(params->seed & 0xffffffffull);
    p.P.seed_hi = (uint32_t)(params->seed >> 32);

    auto take = [&p](size_t n_bytes) {
        const size_t here = p.bytes;
        p.bytes = here + (n_bytes + 255) / 256 * 256;
        return here;
    };
    const size_t ns = (size_t)p.n_slots, nn = (size_t)n;
    p.tables = take(p.pack.bytes.size());
    p.columns = take(sizeof(float) * 8 * nn);
    p.kind = take(sizeof(int) * ns);
    p.energy = take(sizeof(float) * ns);
    p.pos = take(sizeof(float) * 3 * ns);
    p.dir = take(sizeof(float) * 3 * ns);
    p.weight = take(sizeof(float) * ns);
    p.drop = take(sizeof(double) * (size_t)p.blocks);
    p.counts = take(sizeof(unsigned int) * (size_t)p.slot_blocks);
    p.offsets = take(sizeof(unsigned long long) * (size_t)p.slot_blocks);
    p.totals = take(2 * sizeof(unsigned long long));
    if (host_outputs) p.packed = take(36 * ns + 4 * 256);
    return PMC_OK;
}

#define HEAD_CUDA(call)                                  \
    do {                                                 \
        if ((call) != cudaSuccess) return PMC_ERR_CUDA;  \
    } while (0)

Out slots_of(const Plan& p, char* ws) {
    return Out{(int*)(ws + p.kind), (float*)(ws + p.energy), (float*)(ws + p.pos), (float*)(ws + p.dir),
               (float*)(ws + p.weight)};
}

// Trace the primaries `in` (device) into the workspace's slots and count them.
int trace(Plan& p, char* ws, const In& in, cudaStream_t st) {
    char* t = ws + p.tables;
    HEAD_CUDA(cudaMemcpyAsync(t, p.pack.bytes.data(), p.pack.bytes.size(), cudaMemcpyHostToDevice, st));
    const size_t* at = p.at;
    auto i32 = [&]() { return (const int*)(t + *at++); };
    auto f32 = [&]() { return (const float*)(t + *at++); };
    p.S.kind = i32();
    p.S.z_top = f32();
    p.S.z_bottom = f32();
    p.S.jaw_axis = i32();
    p.S.jaw_neg = f32();
    p.S.jaw_pos = f32();
    p.S.jaw_focused = i32();
    p.S.tip_radius = f32();
    p.S.focused_sides = i32();
    p.S.n_pairs = i32();
    p.S.edges_off = i32();
    p.S.tips_off = i32();
    p.S.leaf_edges = f32();
    p.S.tips_neg = f32();
    p.S.tips_pos = f32();
    p.M.log_total = f32();
    const size_t n_mu = (size_t)p.M.n_rows * p.M.n_table;
    p.M.log_compton = p.M.log_total + (sizeof(float) * n_mu + 15) / 16 * 4;
    const Out slots = slots_of(p, ws);
    HEAD_CUDA(cudaMemsetAsync(slots.kind, 0, sizeof(int) * (size_t)p.n_slots, st));
    presolve_kernel<<<p.blocks, kThreads, 0, st>>>(p.S, p.M, p.P, p.n, in, slots, p.per_primary,
                                                   (double*)(ws + p.drop));
    count_slots<<<p.slot_blocks, kThreads, 0, st>>>(slots.kind, p.n_slots, (unsigned int*)(ws + p.counts));
    unsigned long long* totals = (unsigned long long*)(ws + p.totals);
    pmc::scan_tiles_kernel<<<1, 1024, 0, st>>>((const unsigned int*)(ws + p.counts), p.slot_blocks,
                                               (unsigned long long*)(ws + p.offsets), 1, p.slot_blocks,
                                               (long long*)(totals + 1), totals);
    HEAD_CUDA(cudaGetLastError());
    return PMC_OK;
}

template <bool kNormalize>
int compact(const Plan& p, char* ws, const Out& out, cudaStream_t st) {
    compact_slots<kNormalize><<<p.slot_blocks, kThreads, 0, st>>>(
        slots_of(p, ws), p.n_slots, (const unsigned long long*)(ws + p.offsets),
        (const unsigned long long*)(ws + p.totals), p.n, out);
    HEAD_CUDA(cudaGetLastError());
    return PMC_OK;
}

// The kept count and the dropped weight-energy (summed in block order); waits for st.
int read_totals(const Plan& p, char* ws, int64_t* count, double* dropped, cudaStream_t st) {
    std::vector<double> drop(p.blocks);
    unsigned long long total = 0;
    HEAD_CUDA(cudaMemcpyAsync(drop.data(), ws + p.drop, sizeof(double) * drop.size(), cudaMemcpyDeviceToHost, st));
    HEAD_CUDA(cudaMemcpyAsync(&total, ws + p.totals, sizeof total, cudaMemcpyDeviceToHost, st));
    HEAD_CUDA(cudaStreamSynchronize(st));
    double sum = 0.0;
    for (double v : drop) sum += v;
    if (dropped) *dropped = sum;
    *count = (int64_t)total;
    return PMC_OK;
}

}  // namespace

extern "C" int pmc_presolve_head(const pmc_head_stack* stack, const pmc_head_mu* mu, const pmc_head_params* params,
                                 int64_t n, const float* energy, const float* pos, const float* dir,
                                 const float* weight, int64_t capacity, int32_t* out_kind, float* out_energy,
                                 float* out_pos, float* out_dir, float* out_weight, int64_t* count,
                                 double* dropped) {
    if (!count || n < 1 || !energy || !pos || !dir || !weight || capacity < 0 || !params) return PMC_ERR_INVALID;
    Plan p;
    int rc = make_plan(stack, mu, params, n, !params->outputs_on_device, p);
    if (rc) return rc;
    Arena a;
    char* ws = a.alloc<char>(p.bytes);
    if (!ws) return PMC_ERR_CUDA;
    float* col = (float*)(ws + p.columns);
    const size_t nn = (size_t)n;
    HEAD_CUDA(cudaMemcpy(col, energy, sizeof(float) * nn, cudaMemcpyHostToDevice));
    HEAD_CUDA(cudaMemcpy(col + nn, pos, sizeof(float) * 3 * nn, cudaMemcpyHostToDevice));
    HEAD_CUDA(cudaMemcpy(col + 4 * nn, dir, sizeof(float) * 3 * nn, cudaMemcpyHostToDevice));
    HEAD_CUDA(cudaMemcpy(col + 7 * nn, weight, sizeof(float) * nn, cudaMemcpyHostToDevice));
    rc = trace(p, ws, In{col, col + nn, col + 4 * nn, col + 7 * nn, 3, 1}, nullptr);
    if (!rc) rc = read_totals(p, ws, count, dropped, nullptr);
    if (rc) return rc;
    const size_t total = (size_t)*count;
    if (*count > capacity) return PMC_ERR_CAPACITY;
    if (total == 0) return PMC_OK;
    if (!out_kind || !out_energy || !out_pos || !out_dir || !out_weight) return PMC_ERR_INVALID;
    Out out{out_kind, out_energy, out_pos, out_dir, out_weight};
    if (params->outputs_on_device) {  // straight into the caller's device arrays
        rc = compact<false>(p, ws, out, nullptr);
        return rc ? rc : cudaDeviceSynchronize() == cudaSuccess ? PMC_OK : PMC_ERR_CUDA;
    }
    float* packed = (float*)(ws + p.packed);
    Out dev{(int*)packed, packed + total, packed + 2 * total, packed + 5 * total, packed + 8 * total};
    rc = compact<false>(p, ws, dev, nullptr);
    if (rc) return rc;
    HEAD_CUDA(cudaMemcpy(out_kind, dev.kind, sizeof(int) * total, cudaMemcpyDeviceToHost));
    HEAD_CUDA(cudaMemcpy(out_energy, dev.energy, sizeof(float) * total, cudaMemcpyDeviceToHost));
    HEAD_CUDA(cudaMemcpy(out_pos, dev.pos, sizeof(float) * 3 * total, cudaMemcpyDeviceToHost));
    HEAD_CUDA(cudaMemcpy(out_dir, dev.dir, sizeof(float) * 3 * total, cudaMemcpyDeviceToHost));
    HEAD_CUDA(cudaMemcpy(out_weight, dev.weight, sizeof(float) * total, cudaMemcpyDeviceToHost));
    return PMC_OK;
}

extern "C" int pmc_presolve_workspace(const pmc_head_stack* stack, const pmc_head_mu* mu,
                                      const pmc_head_params* params, int64_t n, int64_t* bytes) {
    if (!bytes) return PMC_ERR_INVALID;
    Plan p;
    const int rc = make_plan(stack, mu, params, n, false, p);
    if (!rc) *bytes = (int64_t)p.bytes;
    return rc;
}

extern "C" int pmc_presolve_head_device(const pmc_head_stack* stack, const pmc_head_mu* mu,
                                        const pmc_head_params* params, int64_t n, const float* columns,
                                        void* workspace, int64_t workspace_bytes, int64_t capacity,
                                        int32_t* out_kind, float* out_energy, float* out_pos, float* out_dir,
                                        float* out_weight, int64_t* count, double* dropped, void* stream) {
    if (!count || !columns || !workspace || !out_kind || !out_energy || !out_pos || !out_dir || !out_weight)
        return PMC_ERR_INVALID;
    Plan p;
    int rc = make_plan(stack, mu, params, n, false, p);
    if (rc) return rc;
    if (workspace_bytes < (int64_t)p.bytes || (reinterpret_cast<uintptr_t>(workspace) & 255)) return PMC_ERR_INVALID;
    char* ws = (char*)workspace;
    cudaStream_t st = (cudaStream_t)stream;
    float* col = (float*)(ws + p.columns);
    HEAD_CUDA(cudaMemcpyAsync(col, columns, sizeof(float) * 8 * (size_t)n, cudaMemcpyHostToDevice, st));
    rc = trace(p, ws, In{col, col + n, col + 4 * n, col + 7 * n, 1, n}, st);
    if (rc) return rc;
    const Out out{out_kind, out_energy, out_pos, out_dir, out_weight};
    const bool fits = capacity >= p.n_slots;  // no need to know the count first
    if (fits) rc = compact<true>(p, ws, out, st);
    if (!rc) rc = read_totals(p, ws, count, dropped, st);
    if (rc || fits) return rc;
    if (*count > capacity) return PMC_ERR_CAPACITY;
    rc = compact<true>(p, ws, out, st);
    return rc ? rc : cudaStreamSynchronize(st) == cudaSuccess ? PMC_OK : PMC_ERR_CUDA;
}
