// The routers of routed experts: float32 logits of every token, the choice, the weights.
//
//   chosen-softmax:  z = W x + b; the `top` largest are chosen (the lowest index wins a tie); weights: softmax over the chosen logits only;
//                    optionally the shared expert's gate sigmoid(w_sg . x)
//   scored:          s = softmax(z) over all outputs, or sigmoid(z) of each alone; choice = s + correction (the correction steers the choice, not
//                    the weights); outputs form `group_count` equal groups of neighbours, a group's score is the sum of its `group_top` largest choice
//                    scores, only outputs of the `group_keep` best groups can be chosen (the lowest group index wins a tie, as the lowest output
//                    index does); weight = s * scale, or (normalize) s / (sum of the chosen s + 1e-20) * scale
//
// Few tokens: a block per token, a warp per output.  The kernel is a chain of latencies (row, norm, products, choice), so a warp requests its first
// weight row before the wait on the kernel in front, and where it norms the float32 residual row itself it also leaves the normed row
// (`rows_out`) for the experts behind it (in decode steps 10 to 11 us before, 5.8 to 8.5 now).
//
// Many tokens in bfloat16: sixteen of them are the rows of an mma.sync tile, and a weight crosses L2 once per tile instead of once per token.
// Logits keep 32-bit weights: each is the exact sum of three bfloat16 parts, whose products with the (bfloat16) inputs are exact and meet in
// one float32 sum.  Eight warps share the contraction, then each makes two tokens' choices.  What bounds it is the chain load -
// product - join - choice; 2,048 tokens of width 1,024 and 16 outputs took 25 us with a block per token and take 12.5 here, 4,096
// tokens and 18 outputs 43 and 18 us.
#include "mma.cuh"

namespace {

struct Routing {
    const float *w, *bias, *gate, *correction;             // bias, gate: chosen-softmax; correction: scored
    int n_out, top, scored, score_kind, normalize, group_count, group_keep, group_top;
    float scale;
};

constexpr int AHEAD = 4;                 // pieces of four weights that a lane holds at a time

// a weight row against the input row in shared memory, summed over a warp: lane i takes the pieces of four values i, i + 64, .. and i + 32, i + 96, ..
// in two chains, in a plain loop unrolled UNROLL times with its loads in front (pieces fetched four at a time behind a bound each: 185 -> 255 us for 2,048
// tokens of width 2,048 and 128 outputs).  `pre`: the row's first AHEAD pieces, requested earlier (null: none)
template <int UNROLL> __device__ __forceinline__ float row_dot(const float* __restrict__ w, const float* __restrict__ x, int n, int lane, const float4* pre) {
    float acc = 0.f, acc1 = 0.f;
    if ((n & 3) == 0 && (reinterpret_cast<uintptr_t>(w) & 15) == 0) {
        const float4* w4 = reinterpret_cast<const float4*>(w);
        const float4* x4 = reinterpret_cast<const float4*>(x);
        auto add = [](float& a, const float4& r, const float4& v) { a = fmaf(r.x, v.x, fmaf(r.y, v.y, fmaf(r.z, v.z, fmaf(r.w, v.w, a)))); };
        const int nv = n / 4;
        int i = lane;
        if (pre) {
#pragma unroll
            for (int j = 0; j < AHEAD; ++j)
                if (lane + 32 * j < nv) add(j & 1 ? acc1 : acc, pre[j], x4[lane + 32 * j]);
            i += 32 * AHEAD;
        }
#pragma unroll UNROLL
        for (; i + 32 < nv; i += 64) {
            const float4 a = __ldg(w4 + i), b = __ldg(w4 + i + 32), xa = x4[i], xb = x4[i + 32];
            add(acc, a, xa);
            add(acc1, b, xb);
        }
        if (i < nv) add(acc, __ldg(w4 + i), x4[i]);
    } else {
        for (int i = lane; i < n; i += 32) acc = fmaf(w[i], x[i], acc);
    }
    return vm_warp_sum(acc + acc1);
}

// the largest of v[0 .. n) over a warp, the lowest index among equals; 0x7fffffff if none is above -inf
__device__ __forceinline__ void arg_max(const float* v, int n, int lane, float& best, int& at) {
    best = -INFINITY;
    at = 0x7fffffff;
    for (int e = lane; e < n; e += 32) {
        const float x = v[e];
        if (x > best) { best = x; at = e; }                // ascending e: the first maximum stays
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float ob = __shfl_xor_sync(0xffffffffu, best, o);
        const int oa = __shfl_xor_sync(0xffffffffu, at, o);
        if (ob > best || (ob == best && oa < at)) { best = ob; at = oa; }
    }
}

__device__ void choose_softmax(float* z, const Routing& r, int lane, int* chosen, float* weight) {
    float first = 0.f, sum = 0.f;
    for (int k = 0; k < r.top; ++k) {
        float best;
        int at;
        arg_max(z, r.n_out, lane, best, at);
        if (at == 0x7fffffff) at = 0;                      // (logits that are no numbers)
        if (k == 0) first = best;
        const float p = expf(best - first);                // the largest chosen logit is the softmax's reference
        sum += p;
        if (lane == 0) {
            chosen[k] = at;
            weight[k] = p;
            z[at] = -INFINITY;
        }
        __syncwarp();
    }
    const float inv = 1.0f / sum;
    for (int k = lane; k < r.top; k += 32) weight[k] *= inv;
}

__device__ void choose_scored(float* sc, float* ch, float* gs, const Routing& r, int lane, int* chosen, float* weight) {
    const int n_out = r.n_out;
    if (r.score_kind == VM_SCORE_SIGMOID) {                // every output scored alone: s = 1 / (1 + exp(-z))
        // Without a correction the order of the scores is the order of the logits, and the logits still tell apart what the sigmoid
        // rounds to the same number (every z above 17 gives 1.0f): the choice is made on z.
        for (int e = lane; e < n_out; e += 32) {
            const float z = sc[e], p = 1.0f / (1.0f + expf(-z));
            sc[e] = p;
            ch[e] = r.correction ? p + r.correction[e] : z;
        }
    } else {
        float mx = -INFINITY;
        for (int e = lane; e < n_out; e += 32) mx = fmaxf(mx, sc[e]);
        mx = vm_warp_max(mx);
        float sum = 0.f;
        for (int e = lane; e < n_out; e += 32) sum += expf(sc[e] - mx);
        sum = vm_warp_sum(sum);
        const float inv = 1.0f / sum;
        for (int e = lane; e < n_out; e += 32) {
            const float p = expf(sc[e] - mx) * inv;
            sc[e] = p;
            ch[e] = p + (r.correction ? r.correction[e] : 0.f);
        }
    }
    __syncwarp();
    if (r.group_count > 1 && r.group_keep < r.group_count) {
        const int per = n_out / r.group_count;
        // a group's score: the sum of its group_top largest scores (1: the largest).  Groups are scored on the scores themselves
        // (with the correction, if any), also where the choice inside them goes by the logits.
        const bool by_logit = r.score_kind == VM_SCORE_SIGMOID && !r.correction;
        for (int g = lane; g < r.group_count; g += 32) {
            float total = 0.f, last = INFINITY;
            int last_at = -1;
            for (int k = 0; k < r.group_top && k < per; ++k) {      // the k-th largest: the largest below (last, last_at) in the order (score descending, index ascending)
                float best = -INFINITY;
                int at = -1;
                for (int i = 0; i < per; ++i) {
                    const float v = by_logit ? sc[g * per + i] : ch[g * per + i];
                    const bool after = v < last || (v == last && i > last_at);
                    if (after && v > best) { best = v; at = i; }
                }
                total += best;
                last = best;
                last_at = at;
            }
            gs[g] = total;
        }
        __syncwarp();
        // a group stays if fewer than group_keep groups come before it in the order (score descending, index ascending)
        for (int g = lane; g < r.group_count; g += 32) {
            int before = 0;
            for (int o = 0; o < r.group_count; ++o) before += (gs[o] > gs[g] || (gs[o] == gs[g] && o < g)) ? 1 : 0;
            if (before >= r.group_keep)
                for (int i = 0; i < per; ++i) ch[g * per + i] = -INFINITY;
        }
        __syncwarp();
    }
    float sum_chosen = 0.f;
    for (int k = 0; k < r.top; ++k) {
        float best;
        int at;
        arg_max(ch, n_out, lane, best, at);
        if (at == 0x7fffffff) at = 0;                      // fewer eligible outputs than `top` (a configuration the host refuses)
        sum_chosen += sc[at];
        if (lane == 0) {
            chosen[k] = at;
            weight[k] = sc[at] * r.scale;
            ch[at] = -INFINITY;
        }
        __syncwarp();
    }
    if (r.normalize) {
        const float inv = r.scale / (sum_chosen + 1e-20f);
        for (int k = lane; k < r.top; k += 32) weight[k] = sc[chosen[k]] * inv;
    }
}

// a block per token.  x: rows in the activation dtype T, or (norm_w given) the float32 residual stream: rmsnorm(x) * norm_w, rounded as T would
// hold it, so that a step gives the same numbers whether the norm ran here or in a kernel of its own.  PER_SM: blocks that an SM holds.  1: up to 32 warps,
// first weights ahead of the wait; 4 and 6: 8 warps, more loads in flight or more blocks (1,024 x 16, 512 tokens 7.0 and 8.2 us, 800 tokens 13.1 and 8.2)
template <typename T, int PER_SM, bool SCORED>
__global__ void __launch_bounds__(PER_SM == 1 ? 1024 : 256, PER_SM)
route_kernel(const void* __restrict__ x, const float* __restrict__ norm_w, float eps, const __grid_constant__ Routing r, int hidden, int* __restrict__ chosen,
             float* __restrict__ weight, float* __restrict__ shared_gate, T* __restrict__ rows_out) {
    __shared__ float red[32];
    extern __shared__ __align__(16) float sm[];            // [hidden] input, [n_out] logits, then scores; scored: [n_out] choice scores, [group_count] group scores
    float* xs = sm;
    float* sc = xs + hidden;
    float* ch = sc + r.n_out;
    float* gs = ch + r.n_out;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5, t = blockIdx.x;
    const int outputs = r.n_out + (r.gate ? 1 : 0);
    auto row = [&](int e) { return e < r.n_out ? r.w + (size_t)e * hidden : r.gate; };
    float4 pre[AHEAD];
    const bool ahead = PER_SM == 1 && warp < outputs && (hidden & 3) == 0 && (reinterpret_cast<uintptr_t>(row(warp)) & 15) == 0;
    if (ahead) {                                           // constants: nothing before this kernel writes them
#pragma unroll
        for (int j = 0; j < AHEAD; ++j)
            if (lane + 32 * j < hidden / 4) pre[j] = reinterpret_cast<const float4*>(row(warp))[lane + 32 * j];
    }
    vm_pdl_launch_dependents();
    vm_pdl_wait();
    if (norm_w == nullptr) {
        const T* from = static_cast<const T*>(x) + (size_t)t * hidden;
        for (int i = threadIdx.x; i < hidden; i += blockDim.x) xs[i] = vm_to_float(from[i]);
    } else {
        const float* from = static_cast<const float*>(x) + (size_t)t * hidden;
        float ss = 0.f;
        for (int i = threadIdx.x; i < hidden; i += blockDim.x) { const float v = from[i]; xs[i] = v; ss += v * v; }
        ss = vm_block_sum(ss, red);
        const float inv = 1.0f / sqrtf(ss / (float)hidden + eps);
        for (int i = threadIdx.x; i < hidden; i += blockDim.x) {
            const T v = vm_from_float<T>(xs[i] * inv * norm_w[i]);
            xs[i] = vm_to_float(v);
            if (rows_out) rows_out[(size_t)t * hidden + i] = v;
        }
    }
    __syncthreads();
    for (int e = warp; e < outputs; e += nw) {
        const float d = row_dot<PER_SM == 1 ? 4 : PER_SM == 4 ? 2 : 1>(row(e), xs, hidden, lane, ahead && e == warp ? pre : nullptr);
        if (lane == 0) {
            if (e < r.n_out) sc[e] = d + (r.bias ? r.bias[e] : 0.f);
            else shared_gate[t] = 1.0f / (1.0f + expf(-d));
        }
    }
    __syncthreads();
    if (warp != 0) return;
    if (SCORED) choose_scored(sc, ch, gs, r, lane, chosen + (size_t)t * r.top, weight + (size_t)t * r.top);
    else choose_softmax(sc, r, lane, chosen + (size_t)t * r.top, weight + (size_t)t * r.top);
}

constexpr int TILE = 16;                 // tokens of a block
constexpr int TILE_WARPS = 8;            // (sixteen left room for one block per SM, and 160 blocks took two turns)
constexpr int MAX_TILES = 8;             // of eight outputs
constexpr int HOLD = 4;                  // blocks of 32 of the contraction whose inputs a warp holds

// eight neighbouring weights as three bfloat16 parts each, in pairs
__device__ __forceinline__ void three_parts(const float4& a, const float4& b, unsigned (&hi)[4], unsigned (&mid)[4], unsigned (&lo)[4]) {
    const float v[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const __nv_bfloat162 h = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
        const float2 hf = __bfloat1622float2(h);
        const float r0 = v[2 * i] - hf.x, r1 = v[2 * i + 1] - hf.y;
        const __nv_bfloat162 m = __floats2bfloat162_rn(r0, r1);
        const float2 mf = __bfloat1622float2(m);
        hi[i] = *reinterpret_cast<const unsigned*>(&h);
        mid[i] = *reinterpret_cast<const unsigned*>(&m);
        lo[i] = vm_pack_bf16(r0 - mf.x, r1 - mf.y);
    }
}

__global__ void __launch_bounds__(TILE_WARPS * 32, 2)
route_tile_kernel(const __nv_bfloat16* __restrict__ x, const __grid_constant__ Routing r, int n_tokens, int hidden, int* __restrict__ chosen, float* __restrict__ weight,
                  float* __restrict__ shared_gate) {
    extern __shared__ __align__(16) float sm[];            // [TILE_WARPS][TILE tokens][columns] partial logits, then per token n_out scores, n_out choice scores, groups
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t4 = lane & 3, t0 = blockIdx.x * TILE;
    const int outputs = r.n_out + (r.gate ? 1 : 0), tiles = (outputs + 7) / 8, cols = tiles * 8 + 2;
    const int blocks = hidden / 32, mine = (blocks + TILE_WARPS - 1) / TILE_WARPS, k0 = warp * mine, k1 = min(blocks, k0 + mine);
    float* scores = sm + (size_t)TILE_WARPS * TILE * cols;
    vm_pdl_launch_dependents();
    vm_pdl_wait();
    float c[MAX_TILES][4];
#pragma unroll
    for (int i = 0; i < MAX_TILES; ++i) c[i][0] = c[i][1] = c[i][2] = c[i][3] = 0.f;
    const uint4 none = make_uint4(0u, 0u, 0u, 0u);
    for (int kb = k0; kb < k1; kb += HOLD) {
        uint4 a[2][HOLD];                                  // tokens g and g + 8: eight neighbouring values are the operands of two products
#pragma unroll
        for (int half = 0; half < 2; ++half)
#pragma unroll
            for (int i = 0; i < HOLD; ++i)
                a[half][i] = kb + i < k1 && t0 + g + 8 * half < n_tokens
                                 ? *reinterpret_cast<const uint4*>(x + (size_t)(t0 + g + 8 * half) * hidden + (kb + i) * 32 + t4 * 8) : none;
#pragma unroll
        for (int n = 0; n < MAX_TILES; ++n) {
            if (n >= tiles) break;
            const int e = n * 8 + g;
            const float* row = (e < r.n_out ? r.w + (size_t)e * hidden : r.gate) + kb * 32 + t4 * 8;
            float4 w[HOLD][2];
#pragma unroll
            for (int i = 0; i < HOLD; ++i)
#pragma unroll
                for (int j = 0; j < 2; ++j)
                    w[i][j] = e < outputs && kb + i < k1 ? *reinterpret_cast<const float4*>(row + i * 32 + 4 * j) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int i = 0; i < HOLD; ++i) {
                unsigned hi[4], mid[4], lo[4];
                three_parts(w[i][0], w[i][1], hi, mid, lo);
                vm_mma_bf16_16816(c[n], a[0][i].x, a[1][i].x, a[0][i].y, a[1][i].y, lo[0], lo[1]);
                vm_mma_bf16_16816(c[n], a[0][i].z, a[1][i].z, a[0][i].w, a[1][i].w, lo[2], lo[3]);
                vm_mma_bf16_16816(c[n], a[0][i].x, a[1][i].x, a[0][i].y, a[1][i].y, mid[0], mid[1]);
                vm_mma_bf16_16816(c[n], a[0][i].z, a[1][i].z, a[0][i].w, a[1][i].w, mid[2], mid[3]);
                vm_mma_bf16_16816(c[n], a[0][i].x, a[1][i].x, a[0][i].y, a[1][i].y, hi[0], hi[1]);
                vm_mma_bf16_16816(c[n], a[0][i].z, a[1][i].z, a[0][i].w, a[1][i].w, hi[2], hi[3]);
            }
        }
    }
    float* part = sm + (size_t)warp * TILE * cols;
#pragma unroll
    for (int n = 0; n < MAX_TILES; ++n) {
        if (n >= tiles) break;
        *reinterpret_cast<float2*>(part + g * cols + n * 8 + 2 * t4) = make_float2(c[n][0], c[n][1]);
        *reinterpret_cast<float2*>(part + (g + 8) * cols + n * 8 + 2 * t4) = make_float2(c[n][2], c[n][3]);
    }
    __syncthreads();
    for (int row = warp; row < TILE && t0 + row < n_tokens; row += TILE_WARPS) {      // a token per warp
        const int t = t0 + row;
        float* sc = scores + (size_t)row * (2 * r.n_out + r.group_count);
        for (int e = lane; e < outputs; e += 32) {
            float d = 0.f;
#pragma unroll
            for (int w = 0; w < TILE_WARPS; ++w) d += sm[(size_t)(w * TILE + row) * cols + e];
            if (e < r.n_out) sc[e] = d + (r.bias ? r.bias[e] : 0.f);
            else shared_gate[t] = 1.0f / (1.0f + expf(-d));
        }
        __syncwarp();
        if (r.scored) choose_scored(sc, sc + r.n_out, sc + 2 * r.n_out, r, lane, chosen + (size_t)t * r.top, weight + (size_t)t * r.top);
        else choose_softmax(sc, r, lane, chosen + (size_t)t * r.top, weight + (size_t)t * r.top);
    }
}

bool aligned16(const void* p) { return reinterpret_cast<uintptr_t>(p) % 16 == 0; }

template <typename T>
int launch_route(const void* x, const float* norm_w, float eps, const Routing& r, int n, int hidden, int* chosen, float* weight, float* shared_gate, void* rows_out,
                 cudaStream_t stream) {
    const size_t smem = (size_t)(r.scored ? hidden + 2 * r.n_out + r.group_count : hidden + r.n_out) * sizeof(float);
    if (smem > 48 * 1024) return VM_ERR_UNSUPPORTED;
    // Sixteen tokens a block once a block per token would be more than the six that an SM holds, or more than three where the weights are 256 KB and more
    // (1,024 x 16: 800 tokens 8.2 us a block per token, 8.6 in tiles, 1,184 tokens 15 and 8.6; 1,024 x 64: 296 tokens 11 and 14.5, 512 tokens 15.5 and 14.5;
    // 2,048 x 64: 296 tokens 20 and 22, 400 tokens 30 and 22)
    const int outputs = r.n_out + (r.gate ? 1 : 0);
    const bool many = n > ((long long)outputs * hidden >= 65536 ? 3 : 6) * vm_sm_count();
    if (sizeof(T) == 2 && !norm_w && many && hidden % 32 == 0 && outputs <= 8 * MAX_TILES && r.group_count <= r.n_out && aligned16(x) && aligned16(r.w) &&
        aligned16(r.gate)) {
        const size_t tile = ((size_t)TILE_WARPS * TILE * ((outputs + 7) / 8 * 8 + 2) + (size_t)TILE * (2 * r.n_out + r.group_count)) * sizeof(float);
        static VmOncePerDevice once;
        const cudaError_t e = vm_allow_smem(once, route_tile_kernel, 100 * 1024);
        if (e != cudaSuccess) return (int)e;
        vm_launch_pdl(route_tile_kernel, dim3((n + TILE - 1) / TILE), dim3(TILE_WARPS * 32), tile, stream, (const __nv_bfloat16*)x, r, n, hidden, chosen, weight, shared_gate);
        return vm_launch_status();
    }
    const int per_sm = n <= vm_sm_count() ? 1 : n <= 4 * vm_sm_count() ? 4 : 6;
    const int threads = per_sm == 1 && r.n_out > 8 ? 1024 : 256;      // few tokens: a warp for each output or two (the block's latency is the step's)
#define VM_ROUTE(P, S)                                                                                                                               \
    if (per_sm == P && (r.scored != 0) == S)                                                                                                         \
        vm_launch_pdl(route_kernel<T, P, S>, dim3(n), dim3(threads), smem, stream, x, norm_w, eps, r, hidden, chosen, weight, shared_gate, (T*)rows_out)
    VM_ROUTE(1, true);
    VM_ROUTE(1, false);
    VM_ROUTE(4, true);
    VM_ROUTE(4, false);
    VM_ROUTE(6, true);
    VM_ROUTE(6, false);
#undef VM_ROUTE
    return vm_launch_status();
}

int route(const void* x, const float* norm_w, float eps, const Routing& r, int n, int hidden, int* chosen, float* weight, float* shared_gate, void* rows_out,
          int act_dtype, cudaStream_t stream) {
    if (rows_out && !norm_w) return VM_ERR_BAD_ARG;
    if (act_dtype == VM_F32) return launch_route<float>(x, norm_w, eps, r, n, hidden, chosen, weight, shared_gate, rows_out, stream);
    if (act_dtype == VM_BF16) return launch_route<__nv_bfloat16>(x, norm_w, eps, r, n, hidden, chosen, weight, shared_gate, rows_out, stream);
    return VM_ERR_UNSUPPORTED;
}

}  // namespace

// chosen int32 [T, top], weight float32 [T, top], shared_gate float32 [T] (written only if w_gate is given); weights, bias and the gate row are
// float32 (exact copies of what the checkpoint stores)
// norm_w given: x is the float32 residual stream and the router norms its rows itself; rows_out (null: none) then receives the normed rows
VM_API int vm_expert_router_rows(const void* x, const float* norm_w, float eps, const float* w_router, const float* b_router, const float* w_gate, int T,
                                 int hidden, int E, int top, int* chosen, float* weight, float* shared_gate, void* rows_out, int act_dtype, cudaStream_t stream) {
    if (T <= 0) return 0;
    if (E <= 0 || top <= 0 || top > E || hidden <= 0) return VM_ERR_BAD_ARG;
    const Routing r{w_router, b_router, w_gate, nullptr, E, top, 0, 0, 0, 1, 1, 1, 1.f};
    return route(x, norm_w, eps, r, T, hidden, chosen, weight, shared_gate, rows_out, act_dtype, stream);
}

VM_API int vm_expert_router(const void* x, const float* norm_w, float eps, const float* w_router, const float* b_router, const float* w_gate, int T,
                            int hidden, int E, int top, int* chosen, float* weight, float* shared_gate, int act_dtype, cudaStream_t stream) {
    return vm_expert_router_rows(x, norm_w, eps, w_router, b_router, w_gate, T, hidden, E, top, chosen, weight, shared_gate, nullptr, act_dtype, stream);
}

// chosen int32 [T, top] (an index >= the number of real experts names an identity expert), weight float32 [T, top]; w_router float32
// [n_out, hidden], correction float32 [n_out] or null; group_count must divide n_out
VM_API int vm_expert_router_scored(const void* x, const float* norm_w, float eps, const float* w_router, const float* correction, int T, int hidden,
                                   int n_out, int top, int group_count, int group_keep, float scale, int* chosen, float* weight, int act_dtype,
                                   cudaStream_t stream) {
    return vm_expert_router_scores(x, norm_w, eps, w_router, correction, T, hidden, n_out, top, group_count, group_keep, scale, VM_SCORE_SOFTMAX, chosen,
                                   weight, act_dtype, stream);
}

// the same with the kind of score as an argument: VM_SCORE_SOFTMAX over all outputs, or VM_SCORE_SIGMOID of each output alone
VM_API int vm_expert_router_scores(const void* x, const float* norm_w, float eps, const float* w_router, const float* correction, int T, int hidden,
                                   int n_out, int top, int group_count, int group_keep, float scale, int score_kind, int* chosen, float* weight,
                                   int act_dtype, cudaStream_t stream) {
    return vm_expert_router_groups(x, norm_w, eps, w_router, correction, T, hidden, n_out, top, group_count, group_keep, 1, scale, score_kind, 0, chosen,
                                   weight, act_dtype, stream);
}

// the same with the number of a group's largest scores whose sum is the group's score
VM_API int vm_expert_router_groups(const void* x, const float* norm_w, float eps, const float* w_router, const float* correction, int T, int hidden,
                                   int n_out, int top, int group_count, int group_keep, int group_top, float scale, int score_kind, int normalize,
                                   int* chosen, float* weight, int act_dtype, cudaStream_t stream) {
    return vm_expert_router_groups_rows(x, norm_w, eps, w_router, correction, T, hidden, n_out, top, group_count, group_keep, group_top, scale, score_kind,
                                        normalize, chosen, weight, nullptr, act_dtype, stream);
}

// the same with rows_out, as vm_expert_router_rows
VM_API int vm_expert_router_groups_rows(const void* x, const float* norm_w, float eps, const float* w_router, const float* correction, int T, int hidden,
                                        int n_out, int top, int group_count, int group_keep, int group_top, float scale, int score_kind, int normalize,
                                        int* chosen, float* weight, void* rows_out, int act_dtype, cudaStream_t stream) {
    if (T <= 0) return 0;
    if (group_top < 1) return VM_ERR_BAD_ARG;
    if (score_kind != VM_SCORE_SOFTMAX && score_kind != VM_SCORE_SIGMOID) return VM_ERR_BAD_ARG;
    if (n_out <= 0 || top <= 0 || hidden <= 0 || group_count <= 0 || n_out % group_count || group_keep <= 0 || group_keep > group_count) return VM_ERR_BAD_ARG;
    if (top > (n_out / group_count) * group_keep) return VM_ERR_BAD_ARG;
    const Routing r{w_router, nullptr, nullptr, correction, n_out, top, 1, score_kind, normalize, group_count, group_keep, group_top, scale};
    return route(x, norm_w, eps, r, T, hidden, chosen, weight, nullptr, rows_out, act_dtype, stream);
}
