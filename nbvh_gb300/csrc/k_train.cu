// k_train.cu -- run-optimisation kernels: training-ray generation and labelling on the device,
// the hash-grid encoding of the training rows, forward + composite loss + backward with the weight
// gradients on the tcgen05 tensor cores (K4 backward), the hash-grid gradient scatter (K3
// backward) and the fused Adam step (K5).
//
// Reference path: NeuralBVHRenderer::render, m_run_optimisation branch
// (src/cuda/neural/neural_bvh_renderer.cu:141-288): granular_sample_bvh_network_input_data
// (src/cuda/neural/neural_bvh_module_kernels.cu:119-264), then tcnn's trainer->training_step
// (encoding + FullyFusedMLP forward, PathTracingCompositeLoss, backward, Adam wrapped in
// ExponentialDecay; configured at src/cuda/neural/neural_bvh_module.cu:118-263).
#include <cuda.h>

#include <cstring>
#include <vector>

#include "device_math.cuh"
#include "net_device.cuh"
#include "nbvh_internal.h"
#include "tc_device.cuh"

namespace nbvh {

namespace {

constexpr unsigned kFull = 0xFFFFFFFFu;

// ---------------------------------------------------------------------------------------------
// Training rays (n_sub_batch = 1): stack_based_sample_uniform_bvh_density
// (include/cuda/neural/neural_bvh_module_common.cuh:703-781), sample_bbox_position (635-660),
// generate_single_bvh_network_output_reference (783-861), LocalT depth target (586-629).
// ---------------------------------------------------------------------------------------------

struct SampleArgs {
    GridParams grid;
    NeuralConsts nc;
    const float4 *neural_nodes;
    TrainCut cut;
    uint32_t neural_fast_div; // neural coordinates in the fast-division domain at every dilation
    const float4 *nodes;
    const float4 *tris;
    const float *albedo;
    float *positions;
    float *targets;
    uint32_t *sample_nodes;
    uint32_t training_step;
    uint32_t batch_size;
    uint32_t n;
    uint32_t learned_lod;
    uint32_t classic_fast_div; // classic BVH coordinates in the fast-division domain
    NodeSurvival survival;
};

__device__ __forceinline__ V3 cube_pos_on_face(int face, float u, float v) // sampling.cuh:85-94
{
    switch (face) {
    case 0: return mk3(1.0f, u, v);
    case 1: return mk3(0.0f, u, v);
    case 2: return mk3(u, 1.0f, v);
    case 3: return mk3(u, 0.0f, v);
    case 4: return mk3(u, v, 1.0f);
    default: return mk3(u, v, 0.0f);
    }
}

// A sample's state after its leaf segment was found: origin | mint, direction | maxt, node | rng |
// dilation.
struct SampleFound {
    float4 o_mint, d_maxt;
    uint4 node_rng;
};

constexpr uint32_t kFindThreads = 256;
constexpr int kFindVisits = 8; // node visits of a traversal between lane refills

// First part of the sampler: every sample's direction, LoD and dilation, then its search for an
// entered leaf segment from random origins in the scaled scene box (a fresh origin after every
// traversal that finds none). Persistent warps take samples from a counter and run the traversals
// in rounds of kFindVisits node visits, refilling the lanes whose sample is done, so that one
// sample's many retries do not hold its warp's other lanes idle. Every sample draws the same
// random numbers in the same order as a thread running it alone.
__global__ void __launch_bounds__(kFindThreads, 4) k_training_find(const __grid_constant__ SampleArgs a,
                                                                  SampleFound *__restrict__ found,
                                                                  uint32_t *__restrict__ counter)
{
    const NeuralConsts &c = a.nc;
    const V3 smin = mk3(c.scene_min[0], c.scene_min[1], c.scene_min[2]);
    const V3 smax = mk3(c.scene_max[0], c.scene_max[1], c.scene_max[2]);
    const float h = __fmul_rn(__fsub_rn(c.sampling_bbox_scaling, 1.0f), 0.5f);
    const int lane = threadIdx.x & 31;
    uint32_t i = 0, rng = 0, sampled_lod = 0, node = 0, guard = 0;
    float dil = 0.f, mint = 0.f, maxt = 0.f;
    V3 o = mk3(0, 0, 0), dir = mk3(0, 0, 0);
    uint32_t stack[kNeuralStackSize];
    int sp = 0;
    RayDiv rdiv;
    bool active = false, need_origin = false, exhausted = false, cull_ok = false;
    for (;;) {
        const unsigned idle = __ballot_sync(0xFFFFFFFFu, !active);
        if (idle != 0u && !exhausted) {
            const int leader = __ffs(idle) - 1;
            uint32_t base = 0;
            if (lane == leader)
                base = atomicAdd(counter, (uint32_t)__popc(idle));
            base = __shfl_sync(0xFFFFFFFFu, base, leader);
            exhausted = base + (uint32_t)__popc(idle) >= a.n;
            const uint32_t k = base + __popc(idle & ((1u << lane) - 1u));
            if (!active && k < a.n) {
                i = k;
                rng = lcg_seed(a.training_step * a.batch_size, 0u, i);
                const float sx = lcg_randomf(rng);
                const float sy = lcg_randomf(rng);
                dir = uniform_sphere(sx, sy);
                // sampled LoD among the ones learned so far (common.cuh:719-721)
                const uint32_t n_lods = kNumBvhLods - a.learned_lod;
                const uint32_t lod_pick = __float2uint_rz(__fmul_rn(lcg_randomf(rng), __uint2float_rn(n_lods)));
                sampled_lod = a.learned_lod + min(lod_pick, n_lods - 1u);
                dil = __fadd_rn(c.fixed_node_dilation, __fmul_rn(lcg_randomf(rng), c.node_extent_dilation));
                mint = maxt = 0.f;
                node = 0;
                guard = 0;
                need_origin = true;
                active = true;
            }
        }
        if (!__any_sync(0xFFFFFFFFu, active)) {
            if (exhausted)
                break;
            continue;
        }
        if (active) {
            if (need_origin) {
                stack[0] = 0;
                sp = 1;
                const float px = lcg_randomf(rng);
                const float py = lcg_randomf(rng);
                const float pz = lcg_randomf(rng);
                V3 ps = sub3(scale3(mk3(px, py, pz), c.sampling_bbox_scaling), mk3(h, h, h));
                o = add3(mul3(ps, sub3(smax, smin)), smin);
                rdiv = make_raydiv(o, dir, a.neural_fast_div != 0u);
                cull_ok = dir.x != 0.0f && dir.y != 0.0f && dir.z != 0.0f;
                need_origin = false;
            }
            const int res = neural_intersect_train(a.cut, sampled_lod, o, rdiv, cull_ok, stack, sp,
                                                   c.learning_mint_epsilon, c.learning_maxt_epsilon, dil, mint, maxt,
                                                   node, kFindVisits);
            if (res != 2) {
                if (res < 0)
                    sp = 0;
                if (res != 1 && ++guard < 100000u) {
                    need_origin = true; // no leaf from this origin: the next attempt draws another
                } else {
                    SampleFound f;
                    f.o_mint = make_float4(o.x, o.y, o.z, mint);
                    f.d_maxt = make_float4(dir.x, dir.y, dir.z, maxt);
                    f.node_rng = make_uint4(node, rng, __float_as_uint(dil), 0u);
                    found[i] = f;
                    active = false;
                }
            }
        }
    }
}

// Second part of the sampler, one thread per sample: leaf-boundary origins, node survival, the
// encoded segment points and the classic-BVH labels.
__global__ void __launch_bounds__(128) k_training_samples(const __grid_constant__ SampleArgs a,
                                                          const SampleFound *__restrict__ found)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.n)
        return;
    const NeuralConsts &c = a.nc;
    const V3 smin = mk3(c.scene_min[0], c.scene_min[1], c.scene_min[2]);
    const V3 smax = mk3(c.scene_max[0], c.scene_max[1], c.scene_max[2]);
    const SampleFound f = found[i];
    V3 o = mk3(f.o_mint.x, f.o_mint.y, f.o_mint.z), d = mk3(f.d_maxt.x, f.d_maxt.y, f.d_maxt.z);
    float mint = f.o_mint.w, maxt = f.d_maxt.w;
    const uint32_t node = f.node_rng.x;
    uint32_t rng = f.node_rng.y;
    const float dil = __uint_as_float(f.node_rng.z);
    if (c.leaf_boundary_sampling_ratio != 0.0f && lcg_randomf(rng) <= c.leaf_boundary_sampling_ratio) {
        int f1 = __float2int_rz(__fmul_rn(lcg_randomf(rng), 6.0f));
        f1 = f1 < 5 ? f1 : 5;
        int f2;
        do {
            f2 = __float2int_rz(__fmul_rn(lcg_randomf(rng), 6.0f));
            f2 = f2 < 5 ? f2 : 5;
        } while (f1 == f2);
        const float u1 = lcg_randomf(rng), v1 = lcg_randomf(rng);
        const V3 lp1 = cube_pos_on_face(f1, u1, v1);
        const float u2 = lcg_randomf(rng), v2 = lcg_randomf(rng);
        const V3 lp2 = cube_pos_on_face(f2, u2, v2);
        NodeBox nb = load_node(a.neural_nodes, node);
        V3 ext = sub3(nb.mx, nb.mn);
        V3 center = add3(nb.mn, scale3(ext, 0.5f));
        V3 next = scale3(ext, __fadd_rn(1.0f, dil));
        V3 nmin = sub3(center, scale3(next, 0.5f));
        V3 entry = add3(nmin, mul3(lp1, next));
        V3 exitp = add3(nmin, mul3(lp2, next));
        o = entry;
        d = normalize3(sub3(exitp, entry));
        mint = 0.0f;
        maxt = length3(sub3(exitp, entry));
    }
    if (a.sample_nodes)
        a.sample_nodes[i] = node;
    if (a.survival.enabled) {
        // node survival (neural_bvh_module_kernels.cu:184-199): a rejected sample leaves its slot's
        // previous input and target in place; its node index is already written
        const uint4 st = reinterpret_cast<const uint4 *>(a.survival.stats)[node];
        const float estimate = tree_cut_heuristic(__uint_as_float(st.x), st.y, st.w);
        const float cur_max = a.survival.max_word ? __uint_as_float(*a.survival.max_word) : 0.0f;
        float kept = fmaxf(a.survival.min_prob, __fdiv_rn(estimate, cur_max));
        if (!(estimate <= cur_max))
            kept = 1.0f;
        if (__fmul_rn(a.survival.scale, kept) < lcg_randomf(rng))
            return;
    }

    // encoded segment points (neural_bvh_module_kernels.cu:10-97)
    const float dilation = __fadd_rn(__fadd_rn(1.0f, c.node_extent_dilation), c.fixed_node_dilation);
    const V3 sext = scale3(sub3(smax, smin), dilation);
    const V3 scenter = scale3(add3(smax, smin), 0.5f);
    const V3 epo = encode_world(ray_at(o, d, mint), scenter, sext);
    const V3 epi = encode_world(ray_at(o, d, maxt), scenter, sext);
    const uint32_t P = a.grid.n_points;
    for (uint32_t k = 0; k < P; k++) {
        V3 p = segment_point(epo, epi, segment_t(k, P, a.grid.segment_distribution, rng));
        float *dst = a.positions + ((size_t)i * P + k) * 3u;
        dst[0] = p.x;
        dst[1] = p.y;
        dst[2] = p.z;
    }

    // labels from the classic BLAS on [mint, maxt]
    float t, u, v;
    uint32_t prim, rec = 0;
    classic_traverse<false>(a.nodes, a.tris, o, d, mint, maxt, t, u, v, prim, &rec, a.classic_fast_div != 0u);
    float4 *tg = reinterpret_cast<float4 *>(a.targets + 8u * (size_t)i);
    if (t != FLT_MAX) {
        const float depth =
            __double2float_rn(__ddiv_rn((double)__fsub_rn(t, mint), __dadd_rn((double)__fsub_rn(maxt, mint), 1e-3)));
        float4 r1 = __ldg(a.tris + 3u * rec + 1u), r2 = __ldg(a.tris + 3u * rec + 2u);
        V3 gn = normalize3(cross3(mk3(r1.x, r1.y, r1.z), mk3(r2.x, r2.y, r2.z)));
        V3 nn = scale3(adds3(gn, 1.0f), 0.5f);
        float ax = 0.9f, ay = 0.9f, az = 0.9f;
        if (a.albedo) {
            ax = a.albedo[3u * prim];
            ay = a.albedo[3u * prim + 1u];
            az = a.albedo[3u * prim + 2u];
        }
        tg[0] = make_float4(1.0f, depth, nn.x, nn.y);
        tg[1] = make_float4(nn.z, ax, ay, az);
    } else {
        tg[0] = make_float4(0.f, 0.f, 0.f, 0.f);
        tg[1] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
}

// ---------------------------------------------------------------------------------------------
// Composite loss: include/cuda/neural/utils/loss_gradient.cuh:25-94,
// include/cuda/neural/utils/pt_composite_loss.cuh:18-123
// ---------------------------------------------------------------------------------------------

__device__ __forceinline__ void loss_and_gradient(int type, float target, float pred, float &loss, float &grad)
{
    switch (type) {
    case NBVH_LOSS_RELATIVE_L2: {
        float diff = pred - target;
        float denom = pred * pred + 1e-2f;
        loss = diff * diff / denom;
        grad = 2.0f * diff / denom;
        break;
    }
    case NBVH_LOSS_RELATIVE_L1: {
        float scale = 1.0f / (fabsf(pred) + 1e-2f);
        float diff = pred - target;
        loss = fabsf(diff) * scale;
        grad = copysignf(scale, diff);
        break;
    }
    case NBVH_LOSS_L1: {
        float diff = pred - target;
        loss = fabsf(diff);
        grad = copysignf(1.0f, diff);
        break;
    }
    case NBVH_LOSS_BCE: {
        const float eps = 1e-5f;
        float p = fminf(fmaxf(pred, eps), 1.0f - eps);
        loss = -(target * logf(p) + (1.0f - target) * logf(1.0f - p));
        grad = -(target - p) / (p - (p * p));
        break;
    }
    case NBVH_LOSS_LOG_L2: {
        float diff = logf(1.0f + pred) - logf(1.0f + target);
        loss = diff * diff;
        grad = 2.0f * diff / (pred + 1.0f);
        break;
    }
    case NBVH_LOSS_L_HALF: {
        float sd = sqrtf(fabsf(pred - target));
        loss = sd;
        grad = 1.0f / (2.0f * sd + 1e-5f);
        break;
    }
    default: {
        float diff = pred - target;
        loss = diff * diff;
        grad = 2.0f * diff;
        break;
    }
    }
}

// loss value (normalised by n_total) and d loss / d output (loss scale applied) of one element
__device__ __forceinline__ void composite_loss(const LossConsts &lc, uint32_t ch, float pred, float target,
                                               float target_vis, float &value, float &grad)
{
    float loss = 0.f, g = 0.f;
    const bool ignore = lc.masking ? (target_vis < 0.5f) : false;
    if (ch == 0) {
        loss_and_gradient(lc.visibility_loss, target, pred, loss, g);
        loss *= lc.visibility_loss_scale;
        g *= lc.visibility_loss_scale;
    } else if (ch == 1 && !ignore) {
        loss_and_gradient(lc.depth_loss, target, pred, loss, g);
        loss *= lc.depth_loss_scale;
        g *= lc.depth_loss_scale;
    } else if (ch >= 2 && ch < 5 && !ignore && lc.learn_normal) {
        if (lc.normal_linear) {
            const float n_length = 0.1f;
            float n_axis = (pred * 2.0f - 1.0f) / n_length;
            float lin = n_axis * 0.5f + 0.5f;
            loss_and_gradient(lc.normal_loss, target, lin, loss, g);
            g *= 1.0f / n_length;
        } else {
            loss_and_gradient(lc.normal_loss, target, pred, loss, g);
        }
        loss *= lc.normal_loss_scale;
        g *= lc.normal_loss_scale;
    } else if (ch >= 5 && ch < 8 && !ignore && lc.learn_albedo) {
        if (lc.albedo_linear) {
            const float n_length = 0.1f;
            float lin = pred / n_length;
            loss_and_gradient(lc.albedo_loss, target, lin, loss, g);
            g *= 1.0f / n_length;
        } else {
            loss_and_gradient(lc.albedo_loss, target, pred, loss, g);
        }
        loss *= lc.albedo_loss_scale;
        g *= lc.albedo_loss_scale;
    }
    value = loss * lc.inv_n_total;
    grad = lc.loss_scale * g * lc.inv_n_total;
}

// ---------------------------------------------------------------------------------------------
// The hash-grid features of explicit rows (training batches, nbvh_network_inference), in the MLP
// precision, into rows of n_inputs halves: one thread per (row, point), the levels in order, 8
// features (LPS levels) per 16-byte store (K3 forward). `split`: the point's levels are spread over
// L / LPS threads instead, one store each; batches too small to fill the GPU otherwise are bound by
// the latency of one thread's gathers, level after level (3,001 rows: 37 -> 15 us). Large batches are
// bound by the L1 (ncu, in place order: its data pipe 70%, its request path to L2 65%, L2 53%); 4-byte stores, sixteen partial sectors a
// point, were the rest of 289 us per 2^18 rows, 222 now; large training batches come in an order that
// brings neighbours together (kRowOrderMin).
// ---------------------------------------------------------------------------------------------
template <uint32_t F>
__global__ void __launch_bounds__(256, 4) k_encode_rows(const __grid_constant__ GridParams grid,
                                                     const uint32_t *__restrict__ table,
                                                     const float *__restrict__ positions, uint32_t n,
                                                     __half *__restrict__ feat, uint32_t bf16_, uint32_t split,
                                                     const uint32_t *__restrict__ order)
{
    constexpr uint32_t LPS = 8u / F;
    const uint32_t P = grid.n_points, L = grid.n_levels, G = split ? L / LPS : 1u, LG = L / G;
    const uint64_t w = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (w >= (uint64_t)n * P * G)
        return;
    uint64_t i = w / G; // (row, point)
    const uint32_t l0 = (uint32_t)(w - i * G) * LG;
    if (order) {
        const uint64_t r = i / P;
        i = (uint64_t)__ldg(order + r) * P + (i - r * P);
    }
    const float *src = positions + i * 3u;
    const V3 pos = mk3(__ldg(src), __ldg(src + 1), __ldg(src + 2));
    const bool bf16 = bf16_ != 0u;
    auto pack16 = [bf16](float lo, float hi) { return bf16 ? pack_bf162(lo, hi) : pack_half2(lo, hi); };
    uint32_t *dst = reinterpret_cast<uint32_t *>(feat) + i * L * (F / 2u);
    if (L % LPS == 0u) { // every point's block of L * F halves starts 16-byte aligned
        for (uint32_t l = l0; l < l0 + LG; l += LPS) {
            uint32_t q[4];
#pragma unroll
            for (uint32_t k = 0; k < LPS; k++) {
                if constexpr (F == 2u) {
                    const float2 f = encode_level<true>(table, grid, l + k, pos);
                    q[k] = pack16(f.x, f.y);
                } else {
                    float f[F];
                    encode_level_wide<F>(table, grid, l + k, pos, f);
#pragma unroll
                    for (uint32_t c = 0; c < F / 2u; c++)
                        q[k * (F / 2u) + c] = pack16(f[2u * c], f[2u * c + 1u]);
                }
            }
            *reinterpret_cast<uint4 *>(dst + l * (F / 2u)) = make_uint4(q[0], q[1], q[2], q[3]);
        }
    } else { // level by level (4 bytes for F = 2, 8 for F = 4; F = 8 never comes here)
        for (uint32_t l = 0; l < L; l++) {
            if constexpr (F == 2u) {
                const float2 f = encode_level<true>(table, grid, l, pos);
                dst[l] = pack16(f.x, f.y);
            } else if constexpr (F == 4u) {
                float f[4];
                encode_level_wide<4>(table, grid, l, pos, f);
                *reinterpret_cast<uint2 *>(dst + 2u * l) = make_uint2(pack16(f[0], f[1]), pack16(f[2], f[3]));
            }
        }
    }
}

cudaError_t encode_rows(const GridParams &grid, const uint32_t *table, const float *positions, uint32_t n,
                        __half *features, bool bf16, int num_sms, cudaStream_t s, const uint32_t *order = nullptr)
{
    const uint32_t lps = 8u / grid.n_features, groups = grid.n_levels / lps;
    const uint64_t points = (uint64_t)n * grid.n_points, lanes = (uint64_t)num_sms * 2048u;
    const bool split = grid.n_levels % lps == 0u && points * groups <= lanes;
    const uint64_t threads = points * (split ? groups : 1u);
    const unsigned blocks = (unsigned)((threads + 255u) / 256u);
    const uint32_t b = bf16 ? 1u : 0u, sp = split ? 1u : 0u;
    if (grid.n_features == 4u)
        k_encode_rows<4><<<blocks, 256, 0, s>>>(grid, table, positions, n, features, b, sp, order);
    else if (grid.n_features == 8u)
        k_encode_rows<8><<<blocks, 256, 0, s>>>(grid, table, positions, n, features, b, sp, order);
    else
        k_encode_rows<2><<<blocks, 256, 0, s>>>(grid, table, positions, n, features, b, sp, order);
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------------------------
// Training forward + composite loss + backward on the tensor cores (K3/K4 backward).
//
// k_encode_rows writes each row's FP16 features; then one CTA per SM (two threads per tile row and
// TMEM lane, a warp that issues the MMAs and one that copies the next tile) runs 128-row tiles through
//   forward   Z_{j+1} = X_j W_j^T for every matrix j (tcgen05, M = 128 rows), the ReLU'd 16-bit
//             activations X_{j+1} written back to shared memory (and their ReLU masks kept in
//             registers), then the sigmoid, the composite loss and dZ_out = dL/dZ_out;
//   backward  for j = H .. 0: dX_j = dZ_{j+1} W_j (W_j read transposed, as an MN-major operand)
//             and dW_j^T += X_j^T dZ_{j+1} over the tile's 128 rows (both operands read
//             transposed from the same shared-memory tiles), then dZ_j = dX_j * (X_j > 0);
//             dX_0, rounded to the MLP precision, goes to global memory for the grid scatter.
// The weight gradients stay in tensor memory, accumulated over all the CTA's tiles, and are written out
// once per CTA at the end; the scatter kernel's first blocks sum them. Every [128 rows][C columns] tile
// lives in shared memory in the K-major core-matrix layout (8-column block c at c * 2,048 bytes, row r
// at r * 16 within it): with M = rows it is a K-major operand (LBO 2,048, SBO 128), with K = rows an
// MN-major one (LBO 128, SBO 2,048). The input tile is copied into that layout 16 bytes at a time.
// ---------------------------------------------------------------------------------------------

constexpr uint32_t kTcRows = 128;
// The chain MMA -> accumulator read -> rounding -> shared-memory tile -> next MMA bounds the kernel, ten
// times per tile (20,000 cycles; the tensor cores need some 5,500 of them). What shortens it, us per 2^18
// rows, 128 inputs, 4 hidden layers: two threads per row with half of its columns, input tiles by cp.async
// and the weight-gradient MMAs under the next epilogue 218 -> 215; MMAs issued from uniform registers
// (tc::elect_one) 188 (waiting for them to be issued hid the rest before); a warp of their own for the
// MMAs, every warp waiting for itself, one barrier per step, the next tile's layer 0 under dX_0's
// epilogue and the targets read ahead 155; a second warp that copies the next tile apart from the steps
// 145 (the MMA warp spent 100 cycles on each 512-byte copy, which the next barrier waited for); the next step's
// descriptors made before the barrier 142. The row warps' stores of dX_0 through shared memory, 64 bytes of 8 rows
// at a time instead of 16 bytes of 32, changed nothing.
constexpr uint32_t kTcRowThreads = 256;               // two per tile row
constexpr uint32_t kTcStepThreads = kTcRowThreads + 32u; // and the warp that issues the MMAs
constexpr uint32_t kTcThreads = kTcStepThreads + 32u;    // and the one that copies the next tile
constexpr uint32_t kColBlock = kTcRows * 16u; // bytes between 8-column blocks of a row tile
constexpr uint32_t kTcAccCols = 128;          // TMEM columns of the current layer's accumulator
constexpr uint32_t kTcTmemCols = 512;
constexpr uint32_t kTcWgColsMax = kTcTmemCols - kTcAccCols;
constexpr uint32_t kTcMaxMatrices = kMaxHiddenLayers + 1u;

struct TrainTcArgs {
    const __half *features; // n x n_inputs
    const __half *wpacked;  // 16-bit matrices in the K-major operand layout, back to back
    uint32_t wbytes;
    uint32_t n_inputs;
    uint32_t n_hidden_layers;
    uint32_t n;
    const float *targets; // n x 8
    LossConsts lc;
    __half *dfeat;        // n x n_inputs gradients of the encoded features (emit launches)
    float *wpart;         // [gridDim.x][n_network] each CTA's weight gradients
    uint32_t n_network;
    float *loss_sum;
    float *sample_loss;   // per row: sum of its output channels' loss values (may be NULL)
    uint32_t *status;     // nonzero when a bounded wait gave up
    uint32_t wg_mask;     // bit j: this launch accumulates the gradient of matrix j
    uint32_t emit;        // this launch writes dfeat, the loss and the per-row losses
    uint32_t min_matrix;  // the backward runs from matrix H down to this one
    // shared-memory offsets (bytes from the 1,024-byte aligned base)
    uint32_t x0_off;                      // two input tile buffers of n_inputs * 256 bytes
    uint32_t x_off[kTcMaxMatrices];       // X_j (j = 1..H): 64-column tile (shared when not in wg_mask)
    uint32_t dz_off[2], dzo_off, bar_off; // dZ_j alternates between two tiles (one where only one fits)
    uint32_t loss_off;                    // [kTcRows] loss of each row's upper four channels
    uint32_t wg_col[kTcMaxMatrices];      // TMEM column of the dW_j^T accumulator
    uint32_t acc0_col;                    // layer 0's accumulator (0: that of the other layers and dX_j)
    uint64_t wait_ns;                     // time limit of the phase waits
    uint32_t stall;                       // failure-path test: wait on an mbarrier nothing arrives at
};

__host__ __device__ constexpr uint32_t tc_w0_bytes(uint32_t n_in) { return kNeurons * n_in * 2u; }
__host__ __device__ constexpr uint32_t tc_hidden_w_bytes() { return kNeurons * kNeurons * 2u; }
// byte offset of matrix j in the packed weights; its output and input widths
__host__ __device__ inline uint32_t tc_w_off(uint32_t j, uint32_t n_in)
{
    return j == 0u ? 0u : tc_w0_bytes(n_in) + (j - 1u) * tc_hidden_w_bytes();
}
__host__ __device__ inline uint32_t tc_n_out(uint32_t j, uint32_t H) { return j < H ? kNeurons : kOutputsPadded; }
__host__ __device__ inline uint32_t tc_n_in(uint32_t j, uint32_t n_in) { return j == 0u ? n_in : kNeurons; }
// FP32 parameter offset of matrix j (row-major [out][in])
__host__ __device__ inline uint32_t tc_param_off(uint32_t j, uint32_t n_in)
{
    return j == 0u ? 0u : kNeurons * n_in + (j - 1u) * kNeurons * kNeurons;
}

// this thread's row of a [128][cols] tile: 16-byte chunk c (columns 8c .. 8c + 7)
__device__ __forceinline__ void store_row_chunks(unsigned char *tile, uint32_t row, const uint32_t *words,
                                                 uint32_t chunks)
{
    for (uint32_t c = 0; c < chunks; c++)
        *reinterpret_cast<uint4 *>(tile + c * kColBlock + row * 16u) =
            make_uint4(words[4u * c], words[4u * c + 1u], words[4u * c + 2u], words[4u * c + 3u]);
}

// The operands of one chain of MMAs (tc::mma_chain): D, A and B with their steps, the instruction
// descriptor and the number of MMAs (0: no chain).
struct TcChain {
    uint64_t a_desc, b_desc;
    uint32_t d, a_step, b_step, idesc, count;
};

template <bool BF16, bool FP8>
__global__ void __launch_bounds__(kTcThreads, 1) k_train_tc(const __grid_constant__ TrainTcArgs a)
{
    using Pr = MlpPrec<BF16>;
    extern __shared__ __align__(1024) unsigned char smem[];
    const uint32_t K0 = a.n_inputs, H = a.n_hidden_layers;
    const uint32_t n_tiles = (a.n + kTcRows - 1u) / kTcRows;
    if (blockIdx.x >= n_tiles)
        return;
    // this thread's tile row (= TMEM lane) and half of its columns; the last two warps have none
    const uint32_t tid = threadIdx.x & (kTcRows - 1u), half = threadIdx.x / kTcRows, warp = tid >> 5;
    const bool issuer = threadIdx.x == 0u;
    const uint32_t role = __shfl_sync(kFull, threadIdx.x >> 5, 0);
    const bool mma_warp = role == kTcRowThreads / 32u; // allocates TMEM, issues the MMAs
    const bool copy_warp = role == kTcStepThreads / 32u;
    // weights, layers 1 to H and backward, one nothing arrives at (failure-path test), end, layer 0, next tile
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem + a.bar_off);
    uint32_t *slot = reinterpret_cast<uint32_t *>(bars + 6);
    float *upper_loss = reinterpret_cast<float *>(smem + a.loss_off);
    const uint32_t base = tc::smem_addr(smem);
    const uint32_t bar_w = tc::smem_addr(&bars[0]), bar_mma = tc::smem_addr(&bars[1]),
                   bar_end = tc::smem_addr(&bars[3]), bar_0 = tc::smem_addr(&bars[4]), bar_x = tc::smem_addr(&bars[5]);
    const uint32_t x0_bytes = K0 * kTcRows * 2u;

    if (mma_warp) {
        tc::tmem_alloc(tc::smem_addr(slot), kTcTmemCols);
        tc::tmem_relinquish();
    }
    if (issuer) {
        for (uint32_t b = 0; b < 6u; b++)
            tc::mbar_init(tc::smem_addr(&bars[b]), 1u);
        tc::mbar_init_fence();
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = *slot;
    const uint32_t lane_off = (32u * warp) << 16; // this warp's TMEM lanes

    // Pieces q0 to q1 of tile t's input rows, 512 bytes each by one warp (zeros past the batch): 8 rows and
    // 4 chunks of 16 bytes, which meet in no shared-memory bank. (As sixteen TMA boxes of 128 x 16 bytes
    // the tile took 9,000 of the 34,000 cycles a tile needed, and its issuing thread with it.)
    const uint32_t chunks = K0 / 8u, pieces = (kTcRows / 8u) * ((chunks + 3u) / 4u);
    auto load_tile = [&](uint32_t t, uint32_t buf, uint32_t q0, uint32_t q1) {
        const uint32_t lane = threadIdx.x & 31u;
#pragma unroll 4
        for (uint32_t q = q0; q < q1; q++) {
            const uint32_t r = 8u * (q & 15u) + (lane >> 2), c = 4u * (q >> 4) + (lane & 3u), row = t * kTcRows + r;
            if (c < chunks)
                tc::copy16_async(base + a.x0_off + buf * x0_bytes + c * kColBlock + r * 16u,
                                 a.features + (size_t)(row < a.n ? row : 0u) * K0 + 8u * c, row < a.n);
        }
    };
    uint32_t t = blockIdx.x;
    if (issuer) {
        tc::mbar_expect_tx(bar_w, a.wbytes);
        for (uint32_t o = 0; o < a.wbytes; o += 16384u)
            tc::bulk_load(base + o, reinterpret_cast<const unsigned char *>(a.wpacked) + o,
                          a.wbytes - o < 16384u ? a.wbytes - o : 16384u, bar_w);
    }
    for (uint32_t q = threadIdx.x >> 5; q < pieces; q += kTcThreads / 32u)
        load_tile(t, 0u, q, q + 1u);
    tc::copy_async_wait();
    tc::fence_async_shared(); // the tile's pieces are read by the MMAs
    bool ok = issuer ? tc::mbar_wait(bar_w, 0u, a.wait_ns) : true;
    if (a.stall && issuer) // nothing ever arrives at this barrier: the wait runs out
        ok = ok && tc::mbar_wait(tc::smem_addr(&bars[2]), 0u, a.wait_ns);
    ok = __syncthreads_and(ok);

    uint32_t ph_mma = 0u, ph_0 = 0u, ph_x = 0u, buf = 0u;
    bool first_tile = true;
    float loss_acc = 0.f;
    // Per step one warp issues the MMAs; the row warps wait for those that the epilogue reads, each thread
    // for itself, and write the tiles of the next step. One barrier ends the step and tells everyone if a
    // wait gave up. The last warp keeps out of the steps: it copies the next tile into the other buffer.
    auto mma_done = [&](uint32_t bar, uint32_t &phase) -> bool {
        const bool r = __all_sync(kFull, tc::mbar_wait(bar, phase, a.wait_ns));
        phase ^= 1u;
        tc::fence_after_sync();
        return r;
    };
    bool fine = ok; // this warp's waits; ok is the block's, from the last barrier
    if (copy_warp) {
        for (; fine && t + gridDim.x < n_tiles; t += gridDim.x, buf ^= 1u) {
            // layer 0's commit covers the MMAs of the tile before, the other buffer's last readers
            if (!(fine = mma_done(bar_0, ph_0)))
                break;
            load_tile(t + gridDim.x, buf ^ 1u, 0u, pieces);
            tc::copy_async_wait();
            tc::fence_async_shared();
            __syncwarp();
            if (tc::elect_one())
                tc::mbar_arrive(bar_x);
        }
        first_tile = !ok; // as for the warps below, which run at least one tile
        t = n_tiles;
    }
    for (; ok && t < n_tiles; t += gridDim.x, buf ^= 1u) {
        const uint32_t x0_addr = base + a.x0_off + buf * x0_bytes;
        auto x_addr = [&](uint32_t j) { return j == 0u ? x0_addr : base + a.x_off[j]; };
        // the MMAs of a step, described before the barrier that starts it
        auto forward_chain = [&](uint32_t j) { // Z_{j+1} = X_j W_j^T
            const uint32_t nout = tc_n_out(j, H), nin = tc_n_in(j, K0);
            TcChain c;
            c.d = tmem + (j == 0u ? a.acc0_col : 0u);
            c.a_desc = tc::smem_desc(x_addr(j), kColBlock, 128u);
            c.a_step = kColBlock / 8u;
            c.b_desc = tc::smem_desc(base + tc_w_off(j, K0), nout * 16u, 128u);
            c.b_step = 2u * nout;
            c.idesc = tc::idesc_f16(kTcRows, nout, BF16);
            c.count = nin / 16u;
            return c;
        };
        auto dz_addr = [&](uint32_t j) { return base + (j > H ? a.dzo_off : a.dz_off[j & 1u]); };
        auto dgrad_chain = [&](uint32_t j) { // dX_j (128 x nin) = dZ_{j+1} (128 x nout) . W_j (nout x nin), W_j MN-major
            const uint32_t nout = tc_n_out(j, H), nin = tc_n_in(j, K0);
            TcChain c;
            c.d = tmem;
            c.a_desc = tc::smem_desc(dz_addr(j + 1u), kColBlock, 128u);
            c.a_step = kColBlock / 8u;
            c.b_desc = tc::smem_desc(base + tc_w_off(j, K0), 128u, nout * 16u);
            c.b_step = 16u;
            c.idesc = tc::idesc_f16_major(kTcRows, nin, BF16, false, true);
            c.count = j > a.min_matrix || (j == 0u && a.emit) ? nout / 16u : 0u;
            return c;
        };
        auto wgrad_chain = [&](uint32_t j) { // dW_j^T (128 x nout; rows >= nin unused) += X_j^T . dZ_{j+1}, K = the 128 rows
            const uint32_t nout = tc_n_out(j, H);
            TcChain c;
            c.d = tmem + a.wg_col[j];
            c.a_desc = tc::smem_desc(x_addr(j), 128u, kColBlock);
            c.a_step = 16u;
            c.b_desc = tc::smem_desc(dz_addr(j + 1u), 128u, kColBlock);
            c.b_step = 16u;
            c.idesc = tc::idesc_f16_major(kTcRows, nout, BF16, true, true);
            c.count = ((a.wg_mask >> j) & 1u) ? kTcRows / 16u : 0u;
            return c;
        };
        auto issue = [&](const TcChain &c, uint32_t accumulate) {
            tc::mma_chain(c.d, c.a_desc, c.a_step, c.b_desc, c.b_step, c.idesc, c.count, accumulate);
        };
        TcChain next = forward_chain(0u), next_w = {};
        const uint32_t row = t * kTcRows + tid;
        const bool valid = row < a.n;
        float4 tgt = make_float4(0.f, 0.f, 0.f, 0.f);
        float target_vis = 0.f;
        if (valid && !mma_warp) { // read here, under the forward layers
            tgt = __ldg(reinterpret_cast<const float4 *>(a.targets + (size_t)row * 8u) + half);
            target_vis = __ldg(a.targets + (size_t)row * 8u);
        }
        uint32_t relu_mask[kTcMaxMatrices]; // bits c and 16 + c: columns 32 * half + 2 c and + 2 c + 1 of X_j's row
        float row_loss = 0.f;
        // ---------------- forward ----------------
        for (uint32_t j = 0; j <= H && ok; j++) {
            const uint32_t acc = tmem + (j == 0u ? a.acc0_col : 0u);
            if (mma_warp) {
                if (j == 0u && !first_tile) // the copy of this tile
                    fine = fine && mma_done(bar_x, ph_x);
                if (fine && tc::elect_one()) {
                    tc::fence_after_sync();
                    issue(next, 0u);
                    tc::mma_commit(j == 0u ? bar_0 : bar_mma);
                }
                __syncwarp();
                if (j < H) {
                    next = forward_chain(j + 1u);
                } else {
                    next = dgrad_chain(H);
                    next_w = wgrad_chain(H);
                }
            } else if (!(fine = fine && (j == 0u ? mma_done(bar_0, ph_0) : mma_done(bar_mma, ph_mma)))) {
                // nothing to read
            } else if (j < H) { // X_{j+1} = relu(Z_{j+1}) in the MLP precision (FP8 mode: E4M3 into hidden matrices)
                uint32_t v[2][16];
#pragma unroll
                for (int q = 0; q < 2; q++)
                    tc::tmem_ld16(acc + lane_off + 32u * half + 16u * q, v[q]);
                tc::tmem_wait_ld();
                uint32_t packed[16];
                const bool quant = FP8 && j + 1u < H;
                uint32_t m = 0u;
#pragma unroll
                for (int c = 0; c < 16; c++) {
                    const float lo = __uint_as_float(v[c >> 3][(2 * c) & 15]);
                    const float hi = __uint_as_float(v[c >> 3][(2 * c + 1) & 15]);
                    const uint32_t p = quant ? fp8_act_relu_half2(lo, hi) : pack_relu<BF16>(lo, hi);
                    packed[c] = p;
                    m |= tc::nonzero_halves<BF16>(p) & (0x00010001u << c);
                }
                relu_mask[j + 1u] = m;
                store_row_chunks(smem + a.x_off[j + 1u] + 4u * half * kColBlock, tid, packed, 4u);
            } else { // sigmoid, composite loss, dZ_out: this thread's four of the row's 8 channels
                uint32_t v[8];
                tc::tmem_ld8(tmem + lane_off, v);
                tc::tmem_wait_ld();
                const float t4[4] = {tgt.x, tgt.y, tgt.z, tgt.w};
                float dz[4], val[4];
#pragma unroll
                for (int c = 0; c < 4; c++) {
                    const float y = 1.0f / (1.0f + expf(-__uint_as_float(half ? v[4 + c] : v[c])));
                    float value = 0.f, gr = 0.f;
                    if (valid) {
                        composite_loss(a.lc, 4u * half + (uint32_t)c, y, t4[c], target_vis, value, gr);
                        gr = Pr::round(gr); // 16-bit output gradient
                    }
                    val[c] = value;
                    dz[c] = gr * y * (1.0f - y); // sigmoid backward
                }
                row_loss = (val[0] + val[1]) + (val[2] + val[3]);
                if (half)
                    upper_loss[tid] = row_loss;
                unsigned char *dzo = smem + a.dzo_off + tid * 16u;
                *reinterpret_cast<uint2 *>(dzo + 8u * half) = make_uint2(Pr::pack(dz[0], dz[1]), Pr::pack(dz[2], dz[3]));
                *reinterpret_cast<uint2 *>(dzo + kColBlock + 8u * half) = make_uint2(0u, 0u); // padding outputs
            }
            tc::fence_async_shared(); // the tile rows written above are read by the next MMAs
            tc::fence_before_sync();
            ok = fine = tc::barrier_and(1u, kTcStepThreads, fine);
        }
        if (ok && half == 0u) {
            row_loss += upper_loss[tid];
            loss_acc += row_loss;
            if (valid && a.emit && a.sample_loss)
                a.sample_loss[row] = row_loss;
        }
        // ---------------- backward ----------------
        for (int jj = (int)H; jj >= (int)a.min_matrix && ok; jj--) {
            const uint32_t j = (uint32_t)jj;
            const bool dgrad = j > a.min_matrix || (j == 0u && a.emit);
            // With two dZ tiles the epilogue only waits for dX_j; dW_j's MMAs run under it. A later commit
            // covers them, so they are done before the next step writes the tile they read (its own
            // commit comes after them), before the next tile overwrites X_j, and at the end.
            const bool overlap = dgrad && a.dz_off[0] != a.dz_off[1];
            const bool last = j == a.min_matrix;
            if (mma_warp) {
                if (tc::elect_one()) {
                    tc::fence_after_sync();
                    issue(next, 0u);
                    if (overlap)
                        tc::mma_commit(bar_mma);
                    issue(next_w, first_tile ? 0u : 1u);
                    if (dgrad && !overlap)
                        tc::mma_commit(bar_mma);
                }
                __syncwarp();
                if (!last) {
                    next = dgrad_chain(j - 1u);
                    next_w = wgrad_chain(j - 1u);
                }
            } else if (dgrad && !(fine = fine && mma_done(bar_mma, ph_mma))) {
                // nothing to read
            } else if (j >= 1u && j > a.min_matrix) { // dZ_j = dX_j * (X_j > 0), 16-bit
                uint32_t v[2][16];
#pragma unroll
                for (int q = 0; q < 2; q++)
                    tc::tmem_ld16(tmem + lane_off + 32u * half + 16u * q, v[q]);
                tc::tmem_wait_ld();
                const uint32_t m = relu_mask[j];
                uint32_t packed[16];
#pragma unroll
                for (int c = 0; c < 16; c++) {
                    const uint32_t p = Pr::pack(__uint_as_float(v[c >> 3][(2 * c) & 15]),
                                                __uint_as_float(v[c >> 3][(2 * c + 1) & 15]));
                    packed[c] = p & tc::fill_halves(m << (15 - c));
                }
                store_row_chunks(smem + a.dz_off[j & 1u] + 4u * half * kColBlock, tid, packed, 4u);
            } else if (j == 0u && a.emit) { // dX_0, rounded to the MLP precision, for the grid scatter
                uint4 *dst = reinterpret_cast<uint4 *>(a.dfeat + (size_t)row * K0);
                uint32_t v[4][16]; // 16-column pieces half, half + 2, ...: all in flight, one wait
#pragma unroll
                for (uint32_t i = 0; i < 4u; i++)
                    if (2u * i + half < K0 / 16u) // warp-wide: rows past the batch too
                        tc::tmem_ld16(tmem + lane_off + 16u * (2u * i + half), v[i]);
                tc::tmem_wait_ld();
#pragma unroll
                for (uint32_t i = 0; i < 4u; i++) {
                    const uint32_t q = 2u * i + half;
                    if (valid && q < K0 / 16u) {
                        uint32_t w[8];
#pragma unroll
                        for (int c = 0; c < 8; c++)
                            w[c] = Pr::pack(__uint_as_float(v[i][2 * c]), __uint_as_float(v[i][2 * c + 1]));
                        dst[2u * q] = make_uint4(w[0], w[1], w[2], w[3]);
                        dst[2u * q + 1u] = make_uint4(w[4], w[5], w[6], w[7]);
                    }
                }
            }
            // With an accumulator of its own the next tile's layer 0 runs under dX_0's epilogue; its commit
            // covers this tile's last MMAs.
            if (last && a.acc0_col != 0u)
                break;
            tc::fence_async_shared();
            tc::fence_before_sync();
            ok = fine = tc::barrier_and(1u, kTcStepThreads, fine);
        }
        first_tile = false;
    }
    if (!first_tile) { // the last weight-gradient MMAs
        tc::fence_before_sync();
        ok = __syncthreads_and(fine);
        if (ok) {
            if (mma_warp && tc::elect_one())
                tc::mma_commit(bar_end);
            ok = tc::mbar_wait(bar_end, 0u, a.wait_ns);
            ok = __syncthreads_and(ok);
            tc::fence_after_sync();
        }
    }
    if (!ok) {
        // a wait ran out: record it, give copies and MMAs still in flight one more bounded wait
        tc::copy_async_wait();
        if (issuer)
            tc::mbar_wait(bar_w, 0u);
        for (uint32_t i = threadIdx.x; i < a.n_network; i += kTcThreads) // no gradient of this CTA
            a.wpart[(size_t)blockIdx.x * a.n_network + i] = 0.f;
        if (mma_warp && tc::elect_one()) {
            atomicOr(a.status, 1u);
            tc::mma_commit(bar_end); // covers every MMA issued
            tc::mbar_wait(bar_end, 0u);
        }
    } else if (!first_tile && !mma_warp && !copy_warp) {
        // the CTA's weight gradients: lane m of the dW_j^T accumulator holds column m of dW_j
        for (uint32_t j = 0; j <= H; j++) {
            if (!((a.wg_mask >> j) & 1u))
                continue;
            const uint32_t nout = tc_n_out(j, H), nin = tc_n_in(j, K0);
            float *g = a.wpart + (size_t)blockIdx.x * a.n_network + tc_param_off(j, K0);
            for (uint32_t q = half; q < nout / 16u; q += 2u) {
                uint32_t v[16];
                tc::tmem_ld16(tmem + lane_off + a.wg_col[j] + 16u * q, v);
                tc::tmem_wait_ld();
                if (tid < nin) {
#pragma unroll
                    for (int c = 0; c < 16; c++)
                        g[(size_t)(16u * q + (uint32_t)c) * nin + tid] = __uint_as_float(v[c]);
                }
            }
        }
        if (a.emit) {
#pragma unroll
            for (int off = 16; off > 0; off >>= 1)
                loss_acc += __shfl_xor_sync(kFull, loss_acc, off);
            if ((tid & 31u) == 0u && loss_acc != 0.f)
                atomicAdd(a.loss_sum, loss_acc);
        }
    }
    tc::fence_before_sync();
    __syncthreads();
    if (mma_warp) {
        tc::fence_after_sync();
        tc::tmem_dealloc(tmem, kTcTmemCols);
    }
}

// ---------------------------------------------------------------------------------------------
// Hash-grid gradient scatter (K3 backward): the corners and weights of the forward encoding, each
// corner's feature gradients added with vector atomics (the 16-bit input-feature gradients come from
// k_train_tc). Two neighbouring lanes take one level of one row, the even lane the lower x corners,
// the odd lane the upper ones, and go through the row's points; points in the same cell are summed
// in registers and leave as one set of atomics.
//
// The L2 bounds this kernel: it takes 2e11 32-byte sectors of atomics a second, whatever part of the sector they
// touch (ncu, 2^18 rows at the start of training: 6.72e7 sectors in 327 us, its busiest slice 90% of the time). The points of a row lie on a short segment, so on the coarser levels most
// share a cell (45 sets of corners instead of 64 for the 64 (point, level) pairs of a row). And the
// entries of x and x + 1 lie in one sector 3 times in 4 (2 features; tcnn's hash multiplies x by 1), so
// the two lanes' atomics of one instruction merge into one. Warps are 16 rows of one level: the
// levels' parameters are uniform and a coarse level's warp skips the atomics it merges. 2^18 rows:
// 511 -> 354 us with gradients everywhere (428 with the points merged but one lane for both x
// corners), 352 -> 232 us in a training step of the trained network.
// ---------------------------------------------------------------------------------------------

constexpr uint32_t kScatterThreads = 256, kScatterRows = 32; // rows of a block
// features one thread sums: all of an entry, or 4 of 8
template <uint32_t F>
constexpr uint32_t kScatterFeatures = F < 4u ? F : 4u;

// The weight gradients of k_train_tc's CTAs, which the launch's first blocks sum while the others scatter:
// in FP64 and in CTA order, so that the matrices' gradient is the same in every run (as FP32 atomics of
// 152 CTAs its last bits changed from run to run, and they cost the same time).
struct WeightSum {
    const float *part; // [n_part][n]
    uint32_t n_part, n;
    float *grad;
    uint32_t blocks; // of this launch
};

template <bool BF16, uint32_t F>
__global__ void __launch_bounds__(kScatterThreads) k_grid_scatter(const __grid_constant__ GridParams grid,
                                                                 const __grid_constant__ WeightSum ws,
                                                                 const float *__restrict__ positions,
                                                                 const __half *__restrict__ dfeat, uint32_t n,
                                                                 float *__restrict__ grid_grad, float out_scale)
{
    if (blockIdx.x < ws.blocks) {
        const uint32_t i = blockIdx.x * kScatterThreads + threadIdx.x;
        if (i < ws.n) {
            double sum = 0.0;
#pragma unroll 8
            for (uint32_t k = 0; k < ws.n_part; k++)
                sum += (double)__ldg(ws.part + (size_t)k * ws.n + i);
            ws.grad[i] = (float)sum * out_scale;
        }
        return;
    }
    constexpr uint32_t FT = kScatterFeatures<F>, parts = F / FT;
    const uint32_t P = grid.n_points, L = grid.n_levels;
    for (uint32_t k = threadIdx.x; k < 2u * kScatterRows * L * parts; k += kScatterThreads) {
        const uint32_t up = k & 1u, row = (blockIdx.x - ws.blocks) * kScatterRows + ((k >> 1) & (kScatterRows - 1u));
        const uint32_t lp = k / (2u * kScatterRows), l = lp / parts, part = lp % parts;
        if (row >= n)
            continue;
        const float s = grid.scale[l];
        const uint32_t res = grid.res[l], size = grid.size[l];
        const bool hashed = grid.hashed[l] != 0u;
        float *level = grid_grad + (size_t)grid.offset[l] * F + part * FT;
        float acc[4][FT]; // corners (up, y, z)
        uint32_t cx = 0u, cy = 0u, cz = 0u;
        bool have = false;
        auto flush = [&]() { // adds the sums of cell (cx, cy, cz)
#pragma unroll
            for (uint32_t c = 0; c < 4u; c++) {
                const uint32_t x = cx + up, y = cy + (c & 1u), z = cz + (c >> 1);
                uint32_t i;
                if (hashed) {
                    i = (x ^ (y * 2654435761u) ^ (z * 805459861u)) & (size - 1u);
                } else {
                    i = x + y * res + z * res * res;
                    if (i >= size)
                        i %= size;
                }
                if constexpr (FT == 2u)
                    atomicAdd(reinterpret_cast<float2 *>(level + 2u * (size_t)i), make_float2(acc[c][0], acc[c][1]));
                else
                    atomicAdd(reinterpret_cast<float4 *>(level + (size_t)i * F),
                              make_float4(acc[c][0], acc[c][1], acc[c][2], acc[c][3]));
            }
        };
        const float *src = positions + (size_t)row * P * 3u;
        const uint32_t *gw = reinterpret_cast<const uint32_t *>(dfeat) + ((size_t)row * P * L + l) * (F / 2u) + part * 2u;
        for (uint32_t p = 0; p < P; p++, src += 3, gw += L * (F / 2u)) {
            float g[FT];
            bool any = false;
#pragma unroll
            for (uint32_t q = 0; q < FT / 2u; q++) {
                const float2 v = MlpPrec<BF16>::unpack(__ldg(gw + q));
                g[2u * q] = v.x * out_scale;
                g[2u * q + 1u] = v.y * out_scale;
                any |= v.x != 0.f || v.y != 0.f;
            }
            if (!any)
                continue;
            const float px = __fmaf_rn(__ldg(src), s, 0.5f), py = __fmaf_rn(__ldg(src + 1), s, 0.5f),
                        pz = __fmaf_rn(__ldg(src + 2), s, 0.5f);
            const float flx = floorf(px), fly = floorf(py), flz = floorf(pz);
            const uint32_t gx = (uint32_t)(int32_t)flx, gy = (uint32_t)(int32_t)fly, gz = (uint32_t)(int32_t)flz;
            const float rx = __fsub_rn(px, flx), ry = __fsub_rn(py, fly), rz = __fsub_rn(pz, flz);
            const bool same = have && gx == cx && gy == cy && gz == cz;
            if (have && !same)
                flush();
            cx = gx, cy = gy, cz = gz;
            have = true;
            const float wx = up ? rx : __fsub_rn(1.0f, rx);
#pragma unroll
            for (uint32_t c = 0; c < 4u; c++) {
                const float w = __fmul_rn(__fmul_rn(wx, (c & 1u) ? ry : __fsub_rn(1.0f, ry)),
                                          (c & 2u) ? rz : __fsub_rn(1.0f, rz));
#pragma unroll
                for (uint32_t f = 0; f < FT; f++)
                    acc[c][f] = same ? __fmaf_rn(w, g[f], acc[c][f]) : __fmul_rn(w, g[f]);
            }
        }
        if (have)
            flush();
    }
}

template <bool BF16>
cudaError_t scatter_rows(const GridParams &grid, const WeightSum &ws, const float *positions, const __half *dfeat,
                         uint32_t n, float *grid_grad, float out_scale, cudaStream_t s)
{
    const unsigned blocks = ws.blocks + (n + kScatterRows - 1u) / kScatterRows;
    if (grid.n_features == 4u)
        k_grid_scatter<BF16, 4><<<blocks, kScatterThreads, 0, s>>>(grid, ws, positions, dfeat, n, grid_grad, out_scale);
    else if (grid.n_features == 8u)
        k_grid_scatter<BF16, 8><<<blocks, kScatterThreads, 0, s>>>(grid, ws, positions, dfeat, n, grid_grad, out_scale);
    else
        k_grid_scatter<BF16, 2><<<blocks, kScatterThreads, 0, s>>>(grid, ws, positions, dfeat, n, grid_grad, out_scale);
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------------------------
// K5: Adam + ExponentialDecay (step size precomputed on the host with the bias corrections),
// FP32 master weights, m and v; writes the FP16 copy the kernels read.
// ---------------------------------------------------------------------------------------------

// 16-bit copy of parameter i: the first n_bf16 parameters (the network matrices in BF16 mode) as
// BF16, those in [fp8_lo, fp8_hi) (the hidden 64x64 matrices in FP8 mode) as their FP8-E4M3 value
// at scale 2^6 (exact in FP16), the rest as FP16.
__device__ __forceinline__ __half to_param16(float x, uint32_t i, const ParamPrecision &pp)
{
    if (i < pp.n_bf16) {
        const __nv_bfloat16 b = __float2bfloat16_rn(x);
        return *reinterpret_cast<const __half *>(&b);
    }
    if (i >= pp.fp8_lo && i < pp.fp8_hi)
        return __float2half_rn(__fmul_rn(e4m3_round(__fmul_rn(x, kFp8WeightScale)), 1.0f / kFp8WeightScale));
    return __float2half_rn(x);
}

__global__ void __launch_bounds__(256) k_adam(float *__restrict__ params, __half *__restrict__ params_h,
                                              float *__restrict__ m, float *__restrict__ v,
                                              const float *__restrict__ grad, uint32_t n, float lr_t, float beta1,
                                              float beta2, float eps, float l2_reg, float grad_scale,
                                              const ParamPrecision pp)
{
    const float omb1 = __fsub_rn(1.0f, beta1), omb2 = __fsub_rn(1.0f, beta2);
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float w = params[i];
        const float gr = __fadd_rn(__fmul_rn(grad[i], grad_scale), __fmul_rn(l2_reg, w));
        const float mi = __fadd_rn(__fmul_rn(beta1, m[i]), __fmul_rn(omb1, gr));
        const float vi = __fadd_rn(__fmul_rn(beta2, v[i]), __fmul_rn(omb2, __fmul_rn(gr, gr)));
        m[i] = mi;
        v[i] = vi;
        const float nw = __fsub_rn(w, __fmul_rn(lr_t, __fdiv_rn(mi, __fadd_rn(__fsqrt_rn(vi), eps))));
        params[i] = nw;
        params_h[i] = to_param16(nw, i, pp);
    }
}

__global__ void k_to_half(const float *__restrict__ p, __half *__restrict__ h, uint32_t n, const ParamPrecision pp)
{
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        h[i] = to_param16(p[i], i, pp);
}

__global__ void k_scale(float *__restrict__ p, size_t n, float s)
{
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        p[i] *= s;
}

// One launch of k_train_tc: the matrices whose weight gradients it accumulates (wg_mask), whether
// it also writes the loss and the feature gradients (the launch that reaches matrix 0), and its
// shared-memory layout and TMEM columns.
struct TrainTcPass {
    TrainTcArgs a;
    size_t smem;
};

constexpr size_t kTcSmemLimit = 227u * 1024u;
constexpr size_t kTcSmPerSm = 228u * 1024u;

// Lays out one pass over the matrices in `mask`; false if it does not fit shared memory or TMEM.
bool plan_train_pass(uint32_t n_in, uint32_t H, uint32_t mask, bool emit, TrainTcPass &p)
{
    TrainTcArgs &a = p.a;
    std::memset(&a, 0, sizeof(a));
    const uint32_t wbytes = packed_weight_bytes(n_in, H);
    uint32_t off = (wbytes + 1023u) & ~1023u;
    a.wbytes = wbytes;
    a.x0_off = off;
    off += 2u * n_in * kTcRows * 2u;
    bool transient = false;
    for (uint32_t j = 1; j <= H; j++) {
        if ((mask >> j) & 1u) {
            a.x_off[j] = off;
            off += kNeurons * kTcRows * 2u;
        } else {
            transient = true;
        }
    }
    if (transient) {
        for (uint32_t j = 1; j <= H; j++)
            if (!((mask >> j) & 1u))
                a.x_off[j] = off;
        off += kNeurons * kTcRows * 2u;
    }
    // the weight-gradient MMAs read 128 columns of every X tile (rows past the matrix's input width
    // are ignored): a 64-column tile is always followed by at least 16 KB (the next tile or dZ)
    a.dz_off[0] = a.dz_off[1] = off;
    off += kNeurons * kTcRows * 2u;
    a.dzo_off = off;
    off += kOutputsPadded * kTcRows * 2u;
    a.bar_off = off;
    off += 64u;
    a.loss_off = off;
    off += kTcRows * 4u;
    // a second dZ tile where it fits (1,024-byte tiles first would not change what fits)
    const uint32_t dz2 = (off + 127u) & ~127u;
    if (dz2 + kNeurons * kTcRows * 2u <= kTcSmemLimit) {
        a.dz_off[1] = dz2;
        off = dz2 + kNeurons * kTcRows * 2u;
    }
    uint32_t col = kTcAccCols;
    for (uint32_t j = 0; j <= H; j++) {
        if (!((mask >> j) & 1u))
            continue;
        a.wg_col[j] = col;
        col += tc_n_out(j, H);
    }
    a.acc0_col = col + kNeurons <= kTcTmemCols ? col : 0u;
    if (col > kTcTmemCols || off > kTcSmemLimit)
        return false;
    uint32_t lo = H;
    for (uint32_t j = 0; j <= H; j++)
        if ((mask >> j) & 1u) {
            lo = j;
            break;
        }
    a.wg_mask = mask;
    a.emit = emit ? 1u : 0u;
    a.min_matrix = emit ? 0u : lo;
    // at least half an SM of shared memory, so that one CTA (and its 512 TMEM columns) per SM
    const size_t one_per_sm = kTcSmPerSm / 2u - 1024u + 128u;
    p.smem = off < one_per_sm ? one_per_sm : off;
    return true;
}

// The passes: all matrices in one launch when they fit (up to 5 hidden layers), else groups of
// matrices from the output matrix down, the last group (with matrix 0) writing the loss.
std::vector<TrainTcPass> plan_train_passes(uint32_t n_in, uint32_t H)
{
    std::vector<TrainTcPass> passes;
    TrainTcPass p;
    const uint32_t all = (1u << (H + 1u)) - 1u;
    if (plan_train_pass(n_in, H, all, true, p)) {
        passes.push_back(p);
        return passes;
    }
    uint32_t mask = 0u;
    for (int j = (int)H; j >= 0; j--) {
        const uint32_t trial = mask | (1u << j);
        if (plan_train_pass(n_in, H, trial, j == 0, p)) {
            mask = trial;
            if (j == 0)
                passes.push_back(p);
            continue;
        }
        TrainTcPass done;
        plan_train_pass(n_in, H, mask, false, done);
        passes.push_back(done);
        mask = 1u << j;
        if (j == 0) {
            plan_train_pass(n_in, H, mask, true, p);
            passes.push_back(p);
        }
    }
    return passes;
}

} // namespace

cudaError_t launch_training_samples(const float4 *neural_nodes, const float4 *nodes, const float4 *tris,
                                    const float *albedo, const NeuralConsts &nc, const GridParams &grid,
                                    uint32_t training_step, uint32_t batch_size, uint32_t n, float *positions,
                                    float *targets, uint32_t *sample_nodes, uint32_t learned_lod,
                                    const NodeSurvival *survival, float4 *state, bool classic_fast_div,
                                    const TrainCull &cull, int num_sms, cudaStream_t s)
{
    if (n == 0)
        return cudaSuccess;
    SampleArgs a;
    a.cut = TrainCut{neural_nodes, cull.bounds, cull.grow};
    a.neural_fast_div = cull.fast_div ? 1u : 0u;
    a.grid = grid;
    a.nc = nc;
    a.neural_nodes = neural_nodes;
    a.nodes = nodes;
    a.tris = tris;
    a.albedo = albedo;
    a.positions = positions;
    a.targets = targets;
    a.sample_nodes = sample_nodes;
    a.training_step = training_step;
    a.batch_size = batch_size;
    a.n = n;
    a.learned_lod = learned_lod < kNumBvhLods ? learned_lod : kNumBvhLods - 1u;
    a.classic_fast_div = classic_fast_div ? 1u : 0u;
    if (survival && survival->enabled && survival->stats)
        a.survival = *survival;
    else
        a.survival = NodeSurvival{nullptr, nullptr, 1.0f, 0.0f, 0u};
    SampleFound *found = reinterpret_cast<SampleFound *>(state);
    uint32_t *counter = reinterpret_cast<uint32_t *>(found + n);
    cudaError_t e = cudaMemsetAsync(counter, 0, sizeof(uint32_t), s);
    if (e != cudaSuccess)
        return e;
    uint32_t blocks = (n + kFindThreads - 1u) / kFindThreads;
    if (blocks > (uint32_t)num_sms * 4u)
        blocks = (uint32_t)num_sms * 4u;
    k_training_find<<<blocks, kFindThreads, 0, s>>>(a, found, counter);
    k_training_samples<<<(n + 127u) / 128u, 128, 0, s>>>(a, found);
    return cudaGetLastError();
}

cudaError_t launch_encode_rows(const __half *params_h, const GridParams &grid, uint32_t n_hidden_layers,
                               const float *positions, uint32_t n, __half *features, bool bf16, int num_sms,
                               cudaStream_t s)
{
    if (n == 0)
        return cudaSuccess;
    const uint32_t n_network_params =
        kNeurons * grid.n_inputs + (n_hidden_layers - 1u) * kNeurons * kNeurons + kOutputsPadded * kNeurons;
    const uint32_t *table = reinterpret_cast<const uint32_t *>(params_h + n_network_params);
    return encode_rows(grid, table, positions, n, features, bf16, num_sms, s);
}

// Batches of at least this many rows are encoded in the order of launch_row_order: rows of one place share
// entries of the coarser levels in the L1 (encoding 2^18 random rows 224 -> 172 us). Their gradients are
// scattered in batch order, where neighbours rarely meet on an entry (344 us, 530 in place order). The ordering
// costs some 30 us whatever the batch: gradients of 65,536 rows 286 -> 297 us, 131,072 437 -> 437, 196,608
// 619 -> 608, 262,144 776 -> 754.
constexpr uint32_t kRowOrderMin = 3u << 16;
// order, bins and keys in the buffer of at least 16 halves per row
static_assert((size_t)kRowOrderMin * 32u >= (size_t)kRowOrderMin * 6u + 4u * (kRayBinWords + 4u), "the order fits");

cudaError_t launch_train_step(const __half *params_h, const GridParams &grid, uint32_t n_hidden_layers,
                              const LossConsts &lc, const float *positions, const float *targets, uint32_t n,
                              __half *features, __half *dfeat, __half *wpacked, float *wpart, float *grad,
                              float out_scale, float *loss_sum, bool clear, float *sample_loss, uint32_t *status, bool bf16, bool fp8, int num_sms, cudaStream_t s,
                              uint64_t wait_ns, bool stall, const cudaEvent_t *marks, uint32_t *launches)
{
    if (launches)
        *launches = 0;
    if (n == 0)
        return cudaSuccess;
    cudaError_t e = marks ? cudaEventRecord(marks[0], s) : cudaSuccess;
    if (e != cudaSuccess)
        return e;
    const uint32_t H = n_hidden_layers, n_in = grid.n_inputs;
    const uint32_t n_network_params =
        kNeurons * n_in + (H - 1u) * kNeurons * kNeurons + kOutputsPadded * kNeurons;
    const uint32_t *table = reinterpret_cast<const uint32_t *>(params_h + n_network_params);
    const uint32_t *order = nullptr;
    if (n >= kRowOrderMin) { // the feature gradients are written after the encoding: their buffer holds the order
        uint32_t *words = reinterpret_cast<uint32_t *>(dfeat);
        uint32_t *bins = words + ((size_t)n + 3u) / 4u * 4u;
        e = launch_row_order(positions, n, grid.n_points, reinterpret_cast<uint16_t *>(bins + kRayBinWords), bins, words,
                             num_sms, s);
        if (e != cudaSuccess)
            return e;
        order = words;
    }
    uint32_t count = order ? 5u : 3u; // the order, encoding, packing and scatter
    e = encode_rows(grid, table, positions, n, features, bf16, num_sms, s, order);
    if (e == cudaSuccess)
        e = launch_pack_weights(params_h, n_in, H, wpacked, s, clear ? status : nullptr,
                                clear ? reinterpret_cast<uint32_t *>(loss_sum) : nullptr);
    if (e == cudaSuccess && marks)
        e = cudaEventRecord(marks[1], s);
    if (e != cudaSuccess)
        return e;
    auto kernel = bf16 ? k_train_tc<true, false> : (fp8 ? k_train_tc<false, true> : k_train_tc<false, false>);
    if ((e = allow_max_dynamic_smem(kernel)) != cudaSuccess)
        return e;
    const uint32_t tiles = (n + kTcRows - 1u) / kTcRows;
    const uint32_t blocks = tiles < (uint32_t)num_sms ? tiles : (uint32_t)num_sms;
    for (TrainTcPass &p : plan_train_passes(n_in, H)) {
        TrainTcArgs &a = p.a;
        a.features = features;
        a.wpacked = wpacked;
        a.n_inputs = n_in;
        a.n_hidden_layers = H;
        a.n = n;
        a.targets = targets;
        a.lc = lc;
        a.dfeat = dfeat;
        a.wpart = wpart;
        a.n_network = n_network_params;
        a.loss_sum = loss_sum;
        a.sample_loss = sample_loss;
        a.status = status;
        a.wait_ns = wait_ns ? wait_ns : tc::kWaitLimitNs;
        a.stall = stall ? 1u : 0u;
        kernel<<<blocks, kTcThreads, p.smem, s>>>(a);
        if ((e = cudaGetLastError()) != cudaSuccess)
            return e;
        count++;
    }
    if (marks && (e = cudaEventRecord(marks[2], s)) != cudaSuccess)
        return e;
    const WeightSum ws = {wpart, blocks, n_network_params, grad, (n_network_params + kScatterThreads - 1u) / kScatterThreads};
    e = bf16 ? scatter_rows<true>(grid, ws, positions, dfeat, n, grad + n_network_params, out_scale, s)
             : scatter_rows<false>(grid, ws, positions, dfeat, n, grad + n_network_params, out_scale, s);
    if (e == cudaSuccess && marks)
        e = cudaEventRecord(marks[3], s);
    if (launches)
        *launches = count;
    return e;
}

cudaError_t launch_scale(float *data, size_t n, float scale, cudaStream_t s)
{
    if (n == 0)
        return cudaSuccess;
    k_scale<<<1024, 256, 0, s>>>(data, n, scale);
    return cudaGetLastError();
}

cudaError_t launch_adam(float *params, __half *params_h, float *m, float *v, const float *grad, uint32_t n, float lr_t,
                        float beta1, float beta2, float eps, float l2_reg, float grad_scale, const ParamPrecision &pp,
                        cudaStream_t s)
{
    if (n == 0)
        return cudaSuccess;
    uint32_t blocks = (n + 255u) / 256u;
    if (blocks > 8192u)
        blocks = 8192u;
    k_adam<<<blocks, 256, 0, s>>>(params, params_h, m, v, grad, n, lr_t, beta1, beta2, eps, l2_reg, grad_scale, pp);
    return cudaGetLastError();
}

cudaError_t launch_params_to_half(const float *params, __half *params_h, uint32_t n, const ParamPrecision &pp,
                                  cudaStream_t s)
{
    if (n == 0)
        return cudaSuccess;
    uint32_t blocks = (n + 255u) / 256u;
    if (blocks > 8192u)
        blocks = 8192u;
    k_to_half<<<blocks, 256, 0, s>>>(params, params_h, n, pp);
    return cudaGetLastError();
}

} // namespace nbvh
