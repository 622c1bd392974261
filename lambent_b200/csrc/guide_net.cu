// guide_net.cu - evaluation and training kernels of the learned guiding network (guide_net.cuh) and
// the lam_guide_* entry points.  No counterpart in the reference.
//
//   guide_pack_kernel    f32 master weights -> BF16 core-matrix tiles
//   guide_eval_kernel    128-row tiles: features -> 4 tcgen05 layers -> 40 head outputs per query
//   guide_grad_kernel    forward + backward of 128-row tiles; weight gradients accumulate in TMEM
//                        across the tiles of a CTA and leave as one f32 partial per CTA
//   guide_sum_kernel     sums the partials in a fixed order (deterministic)
//   guide_train_kernel   a run of Adam steps in one cooperative launch: gradients, sums, updates
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "guide_net.cuh"
#include "launch.cuh"
#include "scene.h"
#include "tracer.h"

namespace lam {
namespace net {

constexpr uint32_t ERR_MMA_TIMEOUT = 1u << 8, ERR_MEETING_TIMEOUT = 1u << 9;
// Evaluation: two warpgroups per CTA share the weights; each runs pairs of tiles, tile B's MMAs under tile
// A's epilogue, with its own tiles, barriers and 128 TMEM columns (as the render's sampling kernel does).
constexpr uint32_t EVAL_GROUPS = 2u, EVAL_THREADS = EVAL_GROUPS * TILE;
constexpr uint32_t EVAL_SMEM = LAYERS * LAYER_BYTES + EVAL_GROUPS * 2u * X_BYTES + 64u + 128u;
constexpr uint32_t GRAD_SMEM = LAYERS * LAYER_BYTES + 4u * X_BYTES + G_BYTES + 64u + TILE * LOBES * 4u + 128u;
constexpr uint32_t GRAD_TMEM_COLS = 512;  // acc 0..63, dW[l] at 64 (l + 1)
constexpr uint32_t EVAL_TMEM_COLS = EVAL_GROUPS * 128u;

LAM_DEV uint8_t* align128(uint8_t* p) {
    return reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(p) + 127u) & ~uintptr_t(127));
}

LAM_DEV void stage_weights(uint8_t* W, const uint16_t* packed) {
    const uint4* src = reinterpret_cast<const uint4*>(packed);
    uint4* dst = reinterpret_cast<uint4*>(W);
    for (uint32_t i = threadIdx.x; i < (uint32_t)(LAYERS * LAYER_BYTES / 16); i += blockDim.x) dst[i] = src[i];
}

__global__ void guide_pack_kernel(const float* __restrict__ master, uint16_t* __restrict__ packed) {
    const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= (uint32_t)PARAMS) return;
    const uint32_t l = p / 4096u, o = (p / 64u) % 64u, i = p % 64u;
    const float w = trainable(l, o) ? master[p] : 0.0f;
    __nv_bfloat16 b = __float2bfloat16_rn(w);
    packed[packed_index(l, o, i)] = *reinterpret_cast<uint16_t*>(&b);
}

struct EvalArgs {
    const float* queries;  // n x 9
    uint32_t n;
    float box[6];
    const uint16_t* packed;
    float* out;            // n x 40
    uint32_t* err;
    uint32_t wait_tries;   // polls of each completion wait before it gives up
    uint32_t out_aligned;  // out is a multiple of 16
};

// 100,003 queries: 41 us with one warpgroup and one tile at a time per CTA and 40 separate 4-byte stores per
// row, 22 us here.
__global__ void __launch_bounds__(EVAL_THREADS, 2) guide_eval_kernel(const __grid_constant__ EvalArgs A) {
    extern __shared__ uint8_t smraw[];
    const uint32_t group = threadIdx.x / TILE, row = threadIdx.x & (TILE - 1u);
    uint8_t* W = align128(smraw);
    uint8_t* X[2];
    X[0] = W + LAYERS * LAYER_BYTES + group * 2u * X_BYTES;
    X[1] = X[0] + X_BYTES;
    uint64_t* bars = reinterpret_cast<uint64_t*>(W + LAYERS * LAYER_BYTES + EVAL_GROUPS * 2u * X_BYTES);
    uint32_t* slot = reinterpret_cast<uint32_t*>(bars + 2u * EVAL_GROUPS);
    bars += 2u * group;
    wait_previous();
    stage_weights(W, A.packed);
    if (row == 0) {
        mbar_init(bars);
        mbar_init(bars + 1);
    }
    if (threadIdx.x < 32) tmem_alloc(slot, EVAL_TMEM_COLS);
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = *slot + group * 128u, t_row = tmem + ((row & ~31u) << 16);
    const uint32_t w_addr = smem_u32(W), bar = smem_u32(bars);
    uint32_t phase = 0;
    bool failed = false;
    const uint32_t pairs = (A.n + 2u * TILE - 1u) / (2u * TILE);
    for (uint32_t pair = blockIdx.x * EVAL_GROUPS + group; pair < pairs; pair += gridDim.x * EVAL_GROUPS) {
#pragma unroll
        for (uint32_t h = 0; h < 2u; ++h) {
            const uint32_t idx = (2u * pair + h) * TILE + row;
            Query q{mk(0.0f, 0.0f, 0.0f), mk(0.0f, 1.0f, 0.0f), mk(0.0f, 1.0f, 0.0f)};
            if (idx < A.n) {
                const float* r = A.queries + (size_t)idx * 9u;
                q.pos = mk(r[0], r[1], r[2]);
                q.n = mk(r[3], r[4], r[5]);
                q.wo = mk(r[6], r[7], r[8]);
            }
            float f[WIDTH];
            encode_features(q, A.box, f);
            store_row(X[h], X_RG, row, f);
        }
        bool ok = true;
        for (uint32_t l = 0; l < (uint32_t)LAYERS; ++l) {
            fence_async_smem();
            fence_before();
            if (group_or(group, failed)) {
                failed = true;
                ok = false;
                break;
            }
            if (row == 0) {
                fence_after();
                for (uint32_t h = 0; h < 2u; ++h) {
                    issue_fwd(tmem + 64u * h, smem_u32(X[h]), w_addr + l * LAYER_BYTES);
                    mma_commit(bar + 8u * h);
                }
            }
#pragma unroll
            for (uint32_t h = 0; h < 2u; ++h) {
                if (!mbar_wait(bar + 8u * h, phase, A.wait_tries)) failed = true;
                fence_after();
                if (l < 3u) epilogue_relu(t_row + 64u * h, X[h], row);
            }
            phase ^= 1u;
        }
        if (!ok) break;
#pragma unroll
        for (uint32_t h = 0; h < 2u; ++h) {
            const uint32_t idx = (2u * pair + h) * TILE + row;
            float raw[OUT];
            head_read(t_row + 64u * h, raw);
            if (idx < A.n) {  // rows of 160 bytes; the caller's buffer may be aligned to 4 only
                float* out = A.out + (size_t)idx * OUT;
                if (A.out_aligned) {
#pragma unroll
                    for (int k = 0; k < OUT / 4; ++k)
                        reinterpret_cast<float4*>(out)[k] = make_float4(raw[4 * k], raw[4 * k + 1], raw[4 * k + 2], raw[4 * k + 3]);
                } else {
                    for (int k = 0; k < OUT; ++k) out[k] = raw[k];
                }
            }
        }
    }
    if (failed) {  // let MMAs in flight finish before TMEM is freed
        mbar_wait(bar, phase ^ 1u, DRAIN_TRIES);
        mbar_wait(bar + 8u, phase ^ 1u, DRAIN_TRIES);
    }
    fence_before();
    failed = __syncthreads_or(failed ? 1 : 0) != 0;
    if (failed && threadIdx.x == 0) atomicOr(A.err, ERR_MMA_TIMEOUT);
    if (threadIdx.x < 32) {
        fence_after();
        tmem_free(*slot, EVAL_TMEM_COLS);
    }
}

struct GradArgs {
    const float* recs;      // records, `stride` floats each: pos, normal, wo, wi, weight
    uint32_t stride;
    uint32_t n;             // record count (used when n_dev is null)
    const uint32_t* n_dev;  // device record count, clamped to n
    uint32_t batch;         // rows (multiple of 128)
    uint32_t sequential;    // 1: row b reads record b (rows >= count weigh 0); 0: random records
    uint32_t seed, step;
    float scale;            // loss scale (1 / batch)
    float box[6];
    const uint16_t* packed;
    float* partial;         // gridDim x PARAMS
    float* partial_loss;    // gridDim
    uint32_t* err;
    uint32_t wait_tries;    // polls of each completion wait before it gives up
};

// The gradient kernels run two threads per row of a tile, one per half of its 64 columns (warps w and
// w + 4 reach the same TMEM lanes): with one CTA per SM, encoding, epilogues and stores are chains of
// scalar work with one warp per scheduler to hide them.  The head, whose lobes share their sums, is the
// first half's.
constexpr uint32_t GRAD_THREADS = 2u * TILE;
LAM_DEV uint32_t grad_row() { return threadIdx.x & (TILE - 1u); }
LAM_DEV uint32_t grad_half() { return threadIdx.x / TILE; }

// A CTA's shared memory of the gradient kernels: weights, the inputs of the four layers, the gradient tile.
struct GradSmem {
    uint8_t *W, *X, *G;
    uint64_t* bar;   // [0]: the round that the next epilogue reads; [1]: weight gradients
    uint32_t* slot;
    float* loss;
    float* terms;    // LOBES log terms per row
    LAM_DEV explicit GradSmem(uint8_t* raw) {
        W = align128(raw);
        X = W + LAYERS * LAYER_BYTES;
        G = X + 4 * X_BYTES;
        bar = reinterpret_cast<uint64_t*>(G + G_BYTES);
        slot = reinterpret_cast<uint32_t*>(G + G_BYTES + 16);
        loss = reinterpret_cast<float*>(G + G_BYTES + 20);
        terms = reinterpret_cast<float*>(G + G_BYTES + 64);
    }
    LAM_DEV uint8_t* x(uint32_t l) const { return X + l * X_BYTES; }
};

struct GradCtx : TileCtx {
    uint32_t dw_phase;  // of the weight gradients' barrier
};
// MMAs still in flight after a wait gave up finish before TMEM is read or freed.
LAM_DEV void grad_drain(const GradCtx& c) {
    mbar_wait(c.bar, c.phase ^ 1u, DRAIN_TRIES);
    mbar_wait(c.bar + 8u, c.dw_phase ^ 1u, DRAIN_TRIES);
}

// Clears the gradient tile (its columns 64..127 stay zero), the barrier and the loss; allocates TMEM.
LAM_DEV GradCtx grad_begin(const GradSmem& S, uint32_t wait_tries) {
    uint4* g4 = reinterpret_cast<uint4*>(S.G);
    for (uint32_t i = threadIdx.x; i < G_BYTES / 16u; i += blockDim.x) g4[i] = make_uint4(0u, 0u, 0u, 0u);
    if (threadIdx.x == 0) {
        mbar_init(S.bar);
        mbar_init(S.bar + 1);
        *S.loss = 0.0f;
    }
    if (threadIdx.x < 32) tmem_alloc(S.slot, GRAD_TMEM_COLS);
    fence_before();
    __syncthreads();
    fence_after();
    return GradCtx{{*S.slot, smem_u32(S.bar), 0u, false, wait_tries}, 0u};
}

// Frees TMEM once the CTA's MMAs have finished; reports a wait that gave up.
LAM_DEV void grad_end(const GradCtx& c, uint32_t* err) {
    if (threadIdx.x == 0 && c.failed) atomicOr(err, ERR_MMA_TIMEOUT);
    fence_before();
    __syncthreads();
    if (threadIdx.x < 32) {
        fence_after();
        tmem_free(c.tmem, GRAD_TMEM_COLS);
    }
}

struct GradRecord {
    Query q;
    v3 wi;
    float weight;
};
// The record of this thread's row of a tile.
LAM_DEV GradRecord grad_record(const GradArgs& A, uint32_t n, uint32_t step, uint32_t tile) {
    const uint32_t b = tile * TILE + grad_row();
    bool valid;
    uint32_t idx;
    if (A.sequential) {
        valid = b < n;
        idx = b;
    } else {
        valid = n > 0u;
        idx = valid ? rand_u32(A.seed ^ rand_u32(step * 0x9E3779B9u + b)) % n : 0u;
    }
    GradRecord R{{mk(0.0f, 0.0f, 0.0f), mk(0.0f, 1.0f, 0.0f), mk(0.0f, 1.0f, 0.0f)}, mk(0.0f, 1.0f, 0.0f), 0.0f};
    if (valid) {
        const float* r = A.recs + (size_t)idx * A.stride;
        R.q.pos = mk(r[0], r[1], r[2]);
        R.q.n = mk(r[3], r[4], r[5]);
        R.q.wo = mk(r[6], r[7], r[8]);
        R.wi = mk(r[9], r[10], r[11]);
        R.weight = r[12];
        if (!(R.weight >= 0.0f) || !(R.weight < 3.0e38f)) R.weight = 0.0f;
    }
    return R;
}
LAM_DEV void grad_encode(const GradSmem& S, const GradRecord& R, const float* box) {
    float f[WIDTH];
    // each half computes only the features that it stores
    if (grad_half() == 0u) {
        encode_features(R.q, box, f);
#pragma unroll
        for (uint32_t c = 0; c < 4; ++c) store_chunk(S.x(0), X_RG, grad_row(), c, f + 8 * c);
    } else {
        encode_features(R.q, box, f);
#pragma unroll
        for (uint32_t c = 4; c < 8; ++c) store_chunk(S.x(0), X_RG, grad_row(), c, f + 8 * c);
    }
}

// Forward and backward pass of a tile whose features are in x(0); the weight gradients are added to
// (`add`) or start the TMEM accumulators.  False once a wait has given up.
LAM_DEV bool grad_tile(GradCtx& c, const GradSmem& S, const GradRecord& R, float scale, bool add, float& loss) {
    const uint32_t row = grad_row(), half = grad_half();
    const uint32_t t_row = c.tmem + ((row & ~31u) << 16);
    const uint32_t w_addr = smem_u32(S.W), g_addr = smem_u32(S.G);
    // forward, keeping every layer's input for the backward pass
    for (uint32_t l = 0; l < 4u; ++l) {
        if (!mma_round(c, [&] { issue_fwd(c.tmem, smem_u32(S.x(l)), w_addr + l * LAYER_BYTES); })) return false;
        if (l < 3u) {
            float v[32];
            tmem_ld32(t_row + 32u * half, v);
#pragma unroll
            for (int k = 0; k < 32; ++k) v[k] = fmaxf(v[k], 0.0f);
            if (half) v[31] = 1.0f;  // column 63
#pragma unroll
            for (uint32_t ch = 0; ch < 4; ++ch) store_chunk(S.x(l + 1), X_RG, row, 4u * half + ch, v + 8 * ch);
        } else {
            float raw[OUT], g[OUT / 2];
            head_read(t_row, raw);
            float* terms = S.terms + row * LOBES;
            if (half == 0u) loss += head_grad<0>(raw, R.wi, R.weight, scale, terms, g);
            else head_grad<1>(raw, R.wi, R.weight, scale, terms, g);
#pragma unroll
            for (uint32_t k = 0; k < 8u; ++k)  // outputs 40..63 have no gradient
                *reinterpret_cast<uint2*>(S.G + core_off(row, 8u * k + 4u * half, G_RG)) =
                    k < 5u ? make_uint2(pack_bf16(g[4 * k], g[4 * k + 1]), pack_bf16(g[4 * k + 2], g[4 * k + 3]))
                           : make_uint2(0u, 0u);
        }
    }
    // backward: dW[l] += G^T X[l]; G <- (G W[l]) * relu'(X[l])
    // The input gradients are issued first, with a barrier of their own: their epilogue runs under the
    // weight gradients' MMAs, up to the store into G, which those read.
    for (int l = 3; l >= 0; --l) {
        fence_async_smem();
        fence_before();
        if (__syncthreads_or(c.failed ? 1 : 0)) {
            c.failed = true;
            return false;
        }
        if (threadIdx.x == 0) {
            fence_after();
            if (l > 0) {
                issue_dx(c.tmem, g_addr, w_addr + (uint32_t)l * LAYER_BYTES);
                mma_commit(c.bar);
            }
            issue_dw(c.tmem + 64u * (uint32_t)(l + 1), g_addr, smem_u32(S.x(l)), add);
            mma_commit(c.bar + 8u);
        }
        float v[32];
        if (l > 0) {
            if (!mbar_wait(c.bar, c.phase, c.tries)) c.failed = true;
            c.phase ^= 1u;
            fence_after();
            tmem_ld32(t_row + 32u * half, v);
#pragma unroll
            for (uint32_t ch = 0; ch < 4; ++ch) {
                const uint4 x = load_chunk(S.x(l), X_RG, row, 4u * half + ch);
                const uint32_t xw[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    if (!(bf16_lo(xw[k]) > 0.0f)) v[8 * ch + 2 * k] = 0.0f;
                    if (!(bf16_hi(xw[k]) > 0.0f)) v[8 * ch + 2 * k + 1] = 0.0f;
                }
            }
            if (half) v[31] = 0.0f;  // column 63
        }
        if (!mbar_wait(c.bar + 8u, c.dw_phase, c.tries)) c.failed = true;
        c.dw_phase ^= 1u;
        fence_after();
        if (l > 0) {
#pragma unroll
            for (uint32_t ch = 0; ch < 4; ++ch) store_chunk(S.G, G_RG, row, 4u * half + ch, v + 8 * ch);
        }
    }
    return true;
}

// The CTA's weight-gradient partials: rows 0..63 of each dW accumulator live in the lanes of the first
// two warps of each half.  Partials are stored as 16-byte pieces, [layer][piece of the row][row], so that
// a warp's stores are contiguous (row by row each of them touched 32 lines: 2.2 us of a step).
LAM_DEV void grad_write(const GradCtx& c, float* part, bool any) {
    if (grad_row() < 64u) {
        const uint32_t o = grad_row(), half = grad_half(), t_row = c.tmem + ((o & ~31u) << 16) + 32u * half;
        for (uint32_t l = 0; l < 4u; ++l) {
            float v[32];
            tmem_ld32(t_row + 64u * (l + 1u), v);
            const bool use = any && !c.failed && trainable(l, o);
            float4* dst = reinterpret_cast<float4*>(part) + l * 1024u + 8u * half * 64u + o;
#pragma unroll
            for (int k = 0; k < 8; ++k)
                dst[64 * k] = use ? make_float4(v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    }
}
// The parameter W[l][o][i] at place q of a partial.
LAM_DEV uint32_t partial_param(uint32_t q) {
    const uint32_t l = q / 4096u, piece = (q / 256u) % 16u, o = (q / 4u) % 64u;
    return l * 4096u + o * 64u + 4u * piece + (q & 3u);
}

__global__ void __launch_bounds__(GRAD_THREADS, 1) guide_grad_kernel(const __grid_constant__ GradArgs A) {
    extern __shared__ uint8_t smraw[];
    const GradSmem S(smraw);
    wait_previous();
    stage_weights(S.W, A.packed);
    GradCtx c = grad_begin(S, A.wait_tries);
    uint32_t n = A.n;
    if (A.n_dev) n = min(n, *A.n_dev);
    const uint32_t tiles = A.batch / TILE;
    bool any = false;  // uniform across the CTA
    float loss = 0.0f;
    for (uint32_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const GradRecord R = grad_record(A, n, A.step, tile);
        grad_encode(S, R, A.box);
        if (!grad_tile(c, S, R, A.scale, any, loss)) break;
        any = true;
    }
    // loss: warp sums, then one shared-memory add per warp
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) loss += __shfl_down_sync(0xFFFFFFFFu, loss, o);
    if ((threadIdx.x & 31u) == 0u) atomicAdd(S.loss, loss);
    if (c.failed) grad_drain(c);
    fence_before();
    c.failed = __syncthreads_or(c.failed ? 1 : 0) != 0;
    fence_after();
    grad_write(c, A.partial + (size_t)blockIdx.x * PARAMS, any);
    if (threadIdx.x == 0) A.partial_loss[blockIdx.x] = *S.loss;
    grad_end(c, A.err);
}

struct UpdateArgs {
    const float* partial;
    const float* partial_loss;
    uint32_t parts;
    float* grad;
    float* loss;
    float* master;
    float* m;
    float* v;
    uint16_t* packed;
    float b1, b2, eps;
};

// The sum of the partials' place q, in order; the loads of N are in flight together.  (L2 loads: the
// training kernel reads partials that other SMs wrote while it runs.)
template <uint32_t N>
LAM_DEV float partial_sum(const float* partial, uint32_t parts, uint32_t q) {
    float g = 0.0f;
    uint32_t c = 0;
    for (; c < parts; c += N) {
        float v[N];
#pragma unroll
        for (uint32_t k = 0; k < N; ++k) v[k] = c + k < parts ? __ldcg(partial + (size_t)(c + k) * PARAMS + q) : 0.0f;
#pragma unroll
        for (uint32_t k = 0; k < N; ++k)
            if (c + k < parts) g += v[k];
    }
    return g;
}

// A parameter with its Adam state.
struct AdamState {
    float w, m, v;
};
LAM_DEV AdamState adam_load(const UpdateArgs& A, uint32_t p) { return AdamState{A.master[p], A.m[p], A.v[p]}; }
LAM_DEV void adam_step(const UpdateArgs& A, uint32_t p, AdamState x, float g, float lr_t) {
    const uint32_t l = p / 4096u, o = (p / 64u) % 64u, i = p % 64u;
    if (!trainable(l, o)) return;
    // the contractions are spelled out: left to the compiler they depend on the code around them
    const float m = __fmaf_rn(1.0f - A.b1, g, __fmul_rn(A.b1, x.m));
    const float v = __fmaf_rn(__fmul_rn(1.0f - A.b2, g), g, __fmul_rn(A.b2, x.v));
    A.m[p] = m;
    A.v[p] = v;
    const float w = x.w - lr_t * m / (sqrtf(v) + A.eps);
    A.master[p] = w;
    __nv_bfloat16 b = __float2bfloat16_rn(w);
    A.packed[packed_index(l, o, i)] = *reinterpret_cast<uint16_t*>(&b);
}

// Loss and gradient of a lam_guide_loss_grad: the partials summed in order.
__global__ void guide_sum_kernel(UpdateArgs A) {
    wait_previous();
    const uint32_t q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q == 0) {
        float s = 0.0f;
        for (uint32_t c = 0; c < A.parts; ++c) s += A.partial_loss[c];
        *A.loss = s;
    }
    if (q >= (uint32_t)PARAMS) return;
    const uint32_t p = partial_param(q), l = p / 4096u, o = (p / 64u) % 64u;
    const float g = partial_sum<16>(A.partial, A.parts, q);
    A.grad[p] = trainable(l, o) ? g : 0.0f;
}

// Meetings of all CTAs of the (cooperatively launched) grid, in one word: the arrivals at all meetings so
// far and, above them, 0 or 1 + the meeting that was given up.  A meeting takes place for all CTAs or for
// none, so that an Adam step is taken by all or by none: it is off once that is written before the last
// arrival, and a CTA that stopped waiting, or that cannot go on, writes it by an exchange that fails if
// anyone arrived in between.
enum : uint32_t { MEET_OPEN, MEET_MET, MEET_OFF };
LAM_DEV unsigned long long meet_load(const unsigned long long* word) {
    unsigned long long v;
    asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(word) : "memory");
    return v;
}
LAM_DEV uint32_t meet_state(unsigned long long v, uint32_t k) {
    const uint32_t off = (uint32_t)(v >> 32);  // a meeting after k that is off: all were at k
    if (off) return off - 1u > k ? MEET_MET : MEET_OFF;
    return (uint32_t)v >= (k + 1u) * gridDim.x ? MEET_MET : MEET_OPEN;
}
// Calls meeting k off unless it has taken place; by one thread.  Each exchange that fails follows another
// CTA's arrival or its giving up, at most gridDim.x of them.
LAM_DEV uint32_t meet_give_up(unsigned long long* word, uint32_t k) {
    unsigned long long v = meet_load(word);
    for (uint32_t t = 0; t <= gridDim.x && meet_state(v, k) == MEET_OPEN; ++t) {
        const unsigned long long off = v | ((unsigned long long)(k + 1u) << 32);
        const unsigned long long seen = atomicCAS(word, v, off);
        v = seen == v ? off : seen;
    }
    return meet_state(v, k);
}
LAM_DEV void grid_arrive(unsigned long long* word) {
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        atomicAdd(word, 1ull);
    }
}
// Waits, at most `tries` polls, for the others to arrive at meeting k; false on every thread if it is off.
LAM_DEV bool grid_wait(unsigned long long* word, uint32_t k, uint32_t tries, uint32_t* err) {
    uint32_t state = MEET_MET;
    if (threadIdx.x == 0) {
        state = MEET_OPEN;
        for (uint32_t t = 0; t < tries && state == MEET_OPEN; ++t) state = meet_state(meet_load(word), k);
        if (state == MEET_OPEN) {
            state = meet_give_up(word, k);
            if (state != MEET_MET) atomicOr(err, ERR_MEETING_TIMEOUT);
        }
        __threadfence();
    }
    return __syncthreads_and(state == MEET_MET ? 1 : 0) != 0;
}

// Adam steps A.step .. A.step + steps - 1 in one launch.  Per step a CTA runs its tiles and writes its
// partials; the grid meets; the parameters, spread over all threads, are summed in the partials' order
// (deterministic) and updated; the grid meets again.  Kept between steps: TMEM, the cleared gradient
// tile and the launch; the next step's first records are fetched and encoded while the other CTAs finish
// their partials.  A step of 16,384 records: 18.8 us; as two launches per step,
// 22.5 us of gradients, 5.7 of update and 5 of gaps.  What is left is a chain: weights 2 us, eight MMA rounds
// with their epilogues 7, the head 2.7, partials 1.2, two meetings and the sums 6.
constexpr uint32_t TRAIN_STEPS = 64;  // most steps of a launch
struct TrainArgs {
    GradArgs g;
    UpdateArgs u;
    uint32_t steps;
    unsigned long long* meet;  // zero at launch
    // polls of a meeting; the first one also waits for CTAs that cannot start while other kernels hold their SMs
    uint32_t meet_tries, start_tries;
    float lr[TRAIN_STEPS];
};
__global__ void __launch_bounds__(GRAD_THREADS, 1) guide_train_kernel(const __grid_constant__ TrainArgs T) {
    extern __shared__ uint8_t smraw[];
    const GradSmem S(smraw);
    const GradArgs& A = T.g;
    GradCtx c = grad_begin(S, A.wait_tries);
    uint32_t n = A.n;
    if (A.n_dev) n = min(n, *A.n_dev);
    const uint32_t tiles = A.batch / TILE;
    GradRecord R = grad_record(A, n, A.step, blockIdx.x);
    grad_encode(S, R, A.box);
    for (uint32_t s = 0; s < T.steps; ++s) {
        {
            const uint4* src = reinterpret_cast<const uint4*>(A.packed);
            uint4* dst = reinterpret_cast<uint4*>(S.W);
#pragma unroll
            for (uint32_t k = 0; k < (uint32_t)(LAYERS * LAYER_BYTES / 16) / GRAD_THREADS; ++k)
                dst[k * GRAD_THREADS + threadIdx.x] = __ldcg(src + k * GRAD_THREADS + threadIdx.x);
        }
        float loss = 0.0f;
        bool any = false;
        for (uint32_t tile = blockIdx.x; tile < tiles && !c.failed; tile += gridDim.x) {
            if (any) {
                R = grad_record(A, n, A.step + s, tile);
                grad_encode(S, R, A.box);
            }
            if (!grad_tile(c, S, R, A.scale, any, loss)) break;
            any = true;
        }
        if (c.failed) grad_drain(c);
        fence_before();
        c.failed = __syncthreads_or(c.failed ? 1 : 0) != 0;
        fence_after();
        if (c.failed) {  // no CTA takes this step or another one of this launch
            if (threadIdx.x == 0) meet_give_up(T.meet, 2u * s);
            break;
        }
        grad_write(c, A.partial + (size_t)blockIdx.x * PARAMS, any);
        fence_before();
        grid_arrive(T.meet);
        const bool more = s + 1u < T.steps;
        // under the others' tails: the next step's records, and the state of this thread's first parameter
        if (more) {
            R = grad_record(A, n, A.step + s + 1u, blockIdx.x);
            grad_encode(S, R, A.box);
        }
        const uint32_t q0 = blockIdx.x * TILE + threadIdx.x;
        const bool mine = threadIdx.x < TILE && q0 < (uint32_t)PARAMS;
        AdamState x{0.0f, 0.0f, 0.0f};
        if (mine) x = adam_load(T.u, partial_param(q0));
        if (!grid_wait(T.meet, 2u * s, s ? T.meet_tries : T.start_tries, A.err)) break;
        // 128 parameters per CTA at the grid of a 16,384-record batch
        for (uint32_t q = q0; threadIdx.x < TILE && q < (uint32_t)PARAMS; q += gridDim.x * TILE) {
            const uint32_t p = partial_param(q);
            const float g = partial_sum<64>(A.partial, gridDim.x, q);
            adam_step(T.u, p, q == q0 ? x : adam_load(T.u, p), g, T.lr[s]);
        }
        if (!more) break;
        grid_arrive(T.meet);
        if (!grid_wait(T.meet, 2u * s + 1u, T.meet_tries, A.err)) break;
    }
    grad_end(c, A.err);
}

}  // namespace net

// ---------------------------------------------------------------- host side
static int galloc(lam_guide* g, void** p, size_t bytes) {
    *p = nullptr;
    cudaError_t e = cudaMalloc(p, bytes);
    if (e != cudaSuccess) return cuda_error(e, "cudaMalloc (guide)");
    g->allocs.push_back(*p);
    e = cudaMemset(*p, 0, bytes);
    if (e != cudaSuccess) return cuda_error(e, "cudaMemset (guide)");
    return LAM_OK;
}

static void init_params(uint32_t seed, std::vector<float>& w) {
    // uniform(-a, a) with a = sqrt(6 / fan_in) for the hidden layers and a smaller head; zero biases
    w.assign(net::PARAMS, 0.0f);
    uint64_t s = 0x9E3779B97F4A7C15ull ^ (uint64_t)seed * 0xD1B54A32D192ED03ull;
    auto next = [&]() {
        s ^= s << 13;
        s ^= s >> 7;
        s ^= s << 17;
        return (double)(s >> 11) * (1.0 / 9007199254740992.0);
    };
    for (uint32_t l = 0; l < 4; ++l) {
        const double a = l < 3 ? std::sqrt(6.0 / 64.0) : 0.5 * std::sqrt(6.0 / 64.0);
        for (uint32_t o = 0; o < 64; ++o)
            for (uint32_t i = 0; i < 63; ++i) {
                const double r = (2.0 * next() - 1.0) * a;
                if (net::trainable(l, o)) w[l * 4096 + o * 64 + i] = (float)r;
            }
    }
}

static int upload_params(lam_guide* g, const float* host) {
    cudaError_t e = cudaMemcpy(g->master, host, net::PARAMS * sizeof(float), cudaMemcpyHostToDevice);
    if (e != cudaSuccess) return cuda_error(e, "lam_guide params upload");
    cudaMemset(g->adam_m, 0, net::PARAMS * sizeof(float));
    cudaMemset(g->adam_v, 0, net::PARAMS * sizeof(float));
    net::guide_pack_kernel<<<net::PARAMS / 256, 256>>>(g->master, g->packed);
    e = cudaDeviceSynchronize();
    if (e != cudaSuccess) return cuda_error(e, "lam_guide pack");
    g->steps = 0;
    g->trained_spp = 0;
    return LAM_OK;
}

// CTAs of the gradient kernels: one per tile, at most one per SM.
static uint32_t grad_grid(const lam_guide* g, uint32_t batch) {
    return std::max(1u, std::min<uint32_t>(batch / net::TILE, g->parts));
}

static int setup_kernels(lam_guide* g) {
    if (g->kernels_ready) return LAM_OK;
    cudaError_t e = cudaFuncSetAttribute(net::guide_grad_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, net::GRAD_SMEM);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(net::guide_train_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, net::GRAD_SMEM);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(net::guide_eval_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, net::EVAL_SMEM);
    if (e != cudaSuccess) return cuda_error(e, "guide kernel attributes");
    g->kernels_ready = true;
    return LAM_OK;
}

static void fill_args(lam_guide* g, const float* recs, uint32_t stride, uint32_t n, const uint32_t* n_dev, uint32_t batch,
                      bool sequential, float scale, const float box[6], net::GradArgs& A, net::UpdateArgs& U) {
    A.recs = recs;
    A.stride = stride;
    A.n = n;
    A.n_dev = n_dev;
    A.batch = batch;
    A.sequential = sequential ? 1u : 0u;
    A.seed = g->opts.seed;
    A.step = (uint32_t)g->steps;
    A.scale = scale;
    std::memcpy(A.box, box, sizeof(A.box));
    A.packed = g->packed;
    A.partial = g->partial;
    A.partial_loss = g->partial_loss;
    A.err = g->err;
    A.wait_tries = g->wait_tries;
    U.partial = g->partial;
    U.partial_loss = g->partial_loss;
    U.parts = grad_grid(g, batch);
    U.grad = U.loss = nullptr;
    U.master = g->master;
    U.m = g->adam_m;
    U.v = g->adam_v;
    U.packed = g->packed;
    U.b1 = 0.9f;
    U.b2 = 0.99f;
    U.eps = 1e-8f;
}

// Loss and gradient over n records (two launches).
static int guide_loss_grad(lam_guide* g, const float* recs, uint32_t n, const float box[6], float* grad, float* loss,
                           cudaStream_t st) {
    int rc = setup_kernels(g);
    if (rc) return rc;
    const uint32_t batch = (n + net::TILE - 1) / net::TILE * net::TILE;
    net::GradArgs A;
    net::UpdateArgs U;
    fill_args(g, recs, 13u, n, nullptr, batch, true, 1.0f / (float)n, box, A, U);
    U.grad = grad;
    U.loss = loss;
    Launches go(st);
    go.next(net::guide_grad_kernel, U.parts, net::GRAD_THREADS, net::GRAD_SMEM, A);
    go.next(net::guide_sum_kernel, net::PARAMS / 256, 256, 0, U);
    const cudaError_t e = go.status();
    if (e != cudaSuccess) return cuda_error(e, "guide gradient launch");
    return LAM_OK;
}

// `steps` Adam steps on minibatches of options.batch records drawn from n (or *n_dev, if fewer); counts its
// kernels in *launches.
int guide_train(lam_guide* g, const float* recs, uint32_t stride, uint32_t n, const uint32_t* n_dev, uint32_t steps,
                const float box[6], cudaStream_t st, uint32_t* launches) {
    int rc = setup_kernels(g);
    if (rc) return rc;
    net::TrainArgs T;
    T.meet = reinterpret_cast<unsigned long long*>(g->err + 8);
    // a poll of a meeting is a load that goes to L2; at the default limit of 2^20, some 2 s and 30 s
    T.meet_tries = (uint32_t)std::min<uint64_t>(0xFFFFFFFFull, (uint64_t)g->wait_tries * 4u);
    T.start_tries = (uint32_t)std::min<uint64_t>(0xFFFFFFFFull, (uint64_t)g->wait_tries * 64u);
    while (steps) {
        T.steps = std::min(steps, net::TRAIN_STEPS);
        fill_args(g, recs, stride, n, n_dev, g->opts.batch, false, 1.0f / (float)g->opts.batch, box, T.g, T.u);
        for (uint32_t k = 0; k < T.steps; ++k) {
            const double t = (double)(g->steps + k + 1);
            T.lr[k] = (float)(g->opts.learning_rate * std::sqrt(1.0 - std::pow((double)T.u.b2, t)) /
                              (1.0 - std::pow((double)T.u.b1, t)));
        }
        cudaError_t e = cudaMemsetAsync(T.meet, 0, sizeof(*T.meet), st);
        if (e != cudaSuccess) return cuda_error(e, "guide training");
        void* args[] = {&T};
        // cooperative: the CTAs wait for one another (at most one per SM).  The kernel takes any grid; a smaller one
        // adds the partials of fewer, longer CTAs.
        e = launch_resident(T.u.parts, cudaErrorCooperativeLaunchTooLarge, [&](unsigned grid) {
            const cudaError_t s = cudaLaunchCooperativeKernel((const void*)net::guide_train_kernel, dim3(grid),
                                                              dim3(net::GRAD_THREADS), args, net::GRAD_SMEM, st);
            if (s == cudaErrorCooperativeLaunchTooLarge) (void)cudaGetLastError();
            return s;
        });
        if (e != cudaSuccess) return cuda_error(e, "guide training launch");
        ++*launches;
        g->steps += T.steps;
        steps -= T.steps;
    }
    return LAM_OK;
}

int guide_eval_launch(const lam_guide* g, const float* queries, uint32_t n, const float box[6], float* out,
                      cudaStream_t st) {
    int rc = setup_kernels(const_cast<lam_guide*>(g));
    if (rc) return rc;
    if (n == 0) return LAM_OK;
    net::EvalArgs A;
    A.queries = queries;
    A.n = n;
    std::memcpy(A.box, box, sizeof(A.box));
    A.packed = g->packed;
    A.out = out;
    A.err = g->err;
    A.wait_tries = g->wait_tries;
    A.out_aligned = ((uintptr_t)out & 15u) == 0u ? 1u : 0u;
    const uint32_t per_cta = 2u * net::TILE * net::EVAL_GROUPS;
    const uint32_t grid = std::min<uint32_t>((n + per_cta - 1u) / per_cta, (uint32_t)g->sms * 2u);
    launch_next(net::guide_eval_kernel, grid, net::EVAL_THREADS, net::EVAL_SMEM, st, A);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_error(e, "lam_guide_eval launch");
    return LAM_OK;
}

int guide_check_error(const lam_guide* g) {
    uint32_t h = 0;
    cudaError_t e = cudaMemcpy(&h, g->err, sizeof(h), cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) return cuda_error(e, "lam_guide error flags");
    if (h & (net::ERR_MMA_TIMEOUT | net::ERR_MEETING_TIMEOUT)) {
        // reported once: the flags start clear again for the next kernels
        e = cudaMemset(g->err, 0, sizeof(h));
        if (e != cudaSuccess) return cuda_error(e, "lam_guide error flags");
        return set_error(LAM_ERR_DEVICE_TIMEOUT, h & net::ERR_MMA_TIMEOUT
                                                     ? "guide network: a tensor-core completion wait gave up"
                                                     : "guide training: the wait for the other thread blocks gave up");
    }
    return LAM_OK;
}

}  // namespace lam

using namespace lam;

extern "C" int lam_guide_options_default(lam_guide_options* o) {
    if (!o) return set_error(LAM_ERR_INVALID_ARGUMENT, "null options");
    o->train_spp = 32;
    o->steps_per_wave = 32;
    o->batch = 16384;
    o->record_capacity = 1u << 21;
    o->learning_rate = 2e-3f;
    o->guide_fraction = 0.5f;
    o->seed = 1;
    return LAM_OK;
}

extern "C" int lam_guide_create(const lam_guide_options* o, lam_guide** out) {
    if (!o || !out) return set_error(LAM_ERR_INVALID_ARGUMENT, "lam_guide_create: null argument");
    *out = nullptr;
    if (o->batch == 0 || o->batch % net::TILE != 0) return set_error(LAM_ERR_INVALID_ARGUMENT, "batch must be a positive multiple of 128");
    if (!(o->guide_fraction >= 0.0f && o->guide_fraction < 1.0f))
        return set_error(LAM_ERR_INVALID_ARGUMENT, "guide_fraction must be in [0, 1)");
    if (!(o->learning_rate > 0.0f)) return set_error(LAM_ERR_INVALID_ARGUMENT, "learning_rate must be positive");
    lam_guide* g = new lam_guide();
    g->opts = *o;
    cudaGetDevice(&g->device);
    cudaDeviceGetAttribute(&g->sms, cudaDevAttrMultiProcessorCount, g->device);
    g->parts = (uint32_t)std::max(1, g->sms);
    int rc = 0;
    rc |= galloc(g, (void**)&g->master, net::PARAMS * sizeof(float));
    rc |= galloc(g, (void**)&g->adam_m, net::PARAMS * sizeof(float));
    rc |= galloc(g, (void**)&g->adam_v, net::PARAMS * sizeof(float));
    rc |= galloc(g, (void**)&g->packed, net::PARAMS * sizeof(uint16_t));
    rc |= galloc(g, (void**)&g->partial, (size_t)g->parts * net::PARAMS * sizeof(float));
    rc |= galloc(g, (void**)&g->partial_loss, (size_t)g->parts * sizeof(float));
    rc |= galloc(g, (void**)&g->err, 16 * sizeof(uint32_t));
    if (o->record_capacity) rc |= galloc(g, (void**)&g->records, (size_t)o->record_capacity * GUIDE_RECORD_STRIDE * sizeof(float));
    if (rc) {
        lam_guide_destroy(g);
        return LAM_ERR_CUDA;
    }
    std::vector<float> w;
    init_params(o->seed, w);
    rc = upload_params(g, w.data());
    if (rc) {
        lam_guide_destroy(g);
        return rc;
    }
    *out = g;
    return LAM_OK;
}

extern "C" int lam_guide_destroy(lam_guide* g) {
    if (!g) return LAM_OK;
    for (void* p : g->allocs) cudaFree(p);
    delete g;
    return LAM_OK;
}

extern "C" int lam_guide_get_params(const lam_guide* g, float* params) {
    if (!g || !params) return set_error(LAM_ERR_INVALID_ARGUMENT, "null argument");
    cudaError_t e = cudaMemcpy(params, g->master, net::PARAMS * sizeof(float), cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) return cuda_error(e, "lam_guide_get_params");
    return LAM_OK;
}

extern "C" int lam_guide_set_params(lam_guide* g, const float* params) {
    if (!g || !params) return set_error(LAM_ERR_INVALID_ARGUMENT, "null argument");
    std::vector<float> w(params, params + net::PARAMS);
    for (uint32_t l = 0; l < 4; ++l)
        for (uint32_t o = 0; o < 64; ++o)
            if (!net::trainable(l, o))
                for (uint32_t i = 0; i < 64; ++i) w[l * 4096 + o * 64 + i] = 0.0f;
    return upload_params(g, w.data());
}

extern "C" int lam_guide_eval(const lam_guide* g, const lam_guide_query* queries, uint32_t n, const float box[6],
                              float* outputs, void* stream) {
    if (!g || !box || (n && (!queries || !outputs))) return set_error(LAM_ERR_INVALID_ARGUMENT, "lam_guide_eval: null argument");
    return guide_eval_launch(g, reinterpret_cast<const float*>(queries), n, box, outputs, (cudaStream_t)stream);
}

extern "C" int lam_guide_loss_grad(lam_guide* g, const lam_guide_record* records, uint32_t n, const float box[6],
                                   float* grad, float* loss, void* stream) {
    if (!g || !box || !grad || !loss || (n && !records)) return set_error(LAM_ERR_INVALID_ARGUMENT, "lam_guide_loss_grad: null argument");
    if (n == 0) return set_error(LAM_ERR_INVALID_ARGUMENT, "lam_guide_loss_grad: no records");
    return guide_loss_grad(g, reinterpret_cast<const float*>(records), n, box, grad, loss, (cudaStream_t)stream);
}

extern "C" int lam_guide_train(lam_guide* g, const lam_guide_record* records, uint32_t n, uint32_t steps,
                               const float box[6], void* stream) {
    if (!g || !box || (n && !records)) return set_error(LAM_ERR_INVALID_ARGUMENT, "lam_guide_train: null argument");
    if (!n) return LAM_OK;
    uint32_t launches = 0;
    return guide_train(g, reinterpret_cast<const float*>(records), 13u, n, nullptr, steps, box, (cudaStream_t)stream, &launches);
}

extern "C" int lam_guide_set_wait_limit(lam_guide* g, uint32_t tries) {
    if (!g) return set_error(LAM_ERR_INVALID_ARGUMENT, "null guide");
    g->wait_tries = tries;
    return LAM_OK;
}

extern "C" int lam_guide_progress(const lam_guide* g, uint64_t* steps, uint32_t* trained_spp) {
    if (!g) return set_error(LAM_ERR_INVALID_ARGUMENT, "null guide");
    if (steps) *steps = g->steps;
    if (trained_spp) *trained_spp = g->trained_spp;
    return guide_check_error(g);
}
