// A routed feed-forward (mixture of experts) for few tokens: every token streams the weight rows of ITS experts.  These are the kernels of the
// 32-bit path, of weights kept wider than the activations, and of sizes that routed_experts_tile.cu does not take.
//
//   z = W_router x + b                      float32 logits; the `top` largest are chosen (the lowest index wins a tie)
//   w = softmax over the chosen logits only
//   y = sum_k w_k  W_down[e_k] act(W_up[e_k] x)   (+ s * W_down_shared act(W_up_shared x),  s = sigmoid(w_sg . x))
//
// Two launches behind the router (expert_router.cu): the up-projections with their activation (a warp per four rows of the token's
// virtual matrix [top * ff + ff_shared, hidden]), the down-projections with the weighted sum (a warp per four output columns; the
// experts are added in the order of their rank, so a token's result does not depend on the batch it is in).
// Experts have no biases.  Weights are float32 or bfloat16 (template W), activations float32 or bfloat16 (template T);
// all sums are float32.
#include "common.cuh"

namespace {

__device__ __forceinline__ float expert_act(float z, int kind) {
    if (kind == VM_ACT_RELU_SQUARED) { const float r = fmaxf(z, 0.f); return r * r; }
    if (kind == VM_ACT_GELU_TANH) return 0.5f * z * (1.0f + tanhf(0.7978845608028654f * (z + 0.044715f * z * z * z)));
    return z / (1.0f + expf(-z));
}

// the clamped gated unit: g <- min(g, limit), u <- clamp(u, -limit, limit), g sigmoid(alpha g) (u + 1)
__device__ __forceinline__ float glu_clamped(float g, float u, float limit, float alpha) {
    g = fminf(g, limit);
    u = fminf(fmaxf(u, -limit), limit);
    return g / (1.0f + expf(-alpha * g)) * (u + 1.0f);
}

// R rows at once against the same vector: the rows' loads are independent and in flight together
template <typename W, int R>
__device__ __forceinline__ void warp_dot_rows(const W* const (&w)[R], const float* __restrict__ x, int n, int lane, float (&out)[R]) {
#pragma unroll
    for (int r = 0; r < R; ++r) out[r] = 0.f;
    bool vec = (n & 7) == 0 && sizeof(W) == 2;
#pragma unroll
    for (int r = 0; r < R; ++r) vec = vec && (reinterpret_cast<uintptr_t>(w[r]) & 15) == 0;
    if (vec) {
        for (int i = lane; i < n / 8; i += 32) {
            uint4 p[R];
#pragma unroll
            for (int r = 0; r < R; ++r) p[r] = reinterpret_cast<const uint4*>(w[r])[i];
            float xv[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) xv[k] = x[i * 8 + k];
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const unsigned u[4] = {p[r].x, p[r].y, p[r].z, p[r].w};
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const __nv_bfloat162 b = *reinterpret_cast<const __nv_bfloat162*>(&u[k]);
                    out[r] = fmaf(__low2float(b), xv[2 * k], out[r]);
                    out[r] = fmaf(__high2float(b), xv[2 * k + 1], out[r]);
                }
            }
        }
    } else {
        for (int i = lane; i < n; i += 32) {
            const float xi = x[i];
#pragma unroll
            for (int r = 0; r < R; ++r) out[r] = fmaf(vm_to_float(w[r][i]), xi, out[r]);
        }
    }
#pragma unroll
    for (int r = 0; r < R; ++r) out[r] = vm_warp_sum(out[r]);
}

constexpr int ROWS_PER_WARP = 4;

// A token's input row as float32 in shared memory.  norm_w == nullptr: x is the row in the activation dtype.  Otherwise x is the
// float32 residual stream and the row is rmsnorm(x) * norm_w, rounded as the activation dtype would hold it, so that a step
// gives the same numbers whether the norm ran here or in a kernel of its own.  `red`: 32 floats of shared memory.
template <typename T>
__device__ __forceinline__ void stage_row(const void* __restrict__ x, const float* __restrict__ norm_w, float eps, int t, int hidden, float* xs,
                                          float* red) {
    if (norm_w == nullptr) {
        const T* row = static_cast<const T*>(x) + (size_t)t * hidden;
        for (int i = threadIdx.x; i < hidden; i += blockDim.x) xs[i] = vm_to_float(row[i]);
        __syncthreads();
        return;
    }
    const float* row = static_cast<const float*>(x) + (size_t)t * hidden;
    float ss = 0.f;
    for (int i = threadIdx.x; i < hidden; i += blockDim.x) { const float v = row[i]; xs[i] = v; ss += v * v; }
    ss = vm_block_sum(ss, red);
    const float inv = 1.0f / sqrtf(ss / (float)hidden + eps);
    for (int i = threadIdx.x; i < hidden; i += blockDim.x) xs[i] = vm_to_float(vm_from_float<T>(xs[i] * inv * norm_w[i]));
    __syncthreads();
}

// ------------------------------------------------------------------------------------------------ up-projections
// grid (row tiles, T); a warp per row r of the token's [top * ff + ff_shared] rows.  An act row has `act_cols` columns:
// those rows and, where identity experts exist (E_real < the router's outputs), the token's input row behind them.
// glu: an expert's up matrix is [2 * ff, hidden], gate rows first, and row r is glu_clamped(gate_r . x, up_r . x).
template <typename T, typename W>
__global__ void experts_up_kernel(const void* __restrict__ x, const float* __restrict__ norm_w, float eps, const W* __restrict__ w_up,
                                  const W* __restrict__ w_up_shared, const int* __restrict__ chosen, int hidden, int ff, int ff_shared, int top,
                                  int act_kind, int act_kind_shared, int E_real, int glu, float limit, float alpha, int act_cols,
                                  const float* __restrict__ weight, T* __restrict__ act) {
    extern __shared__ __align__(16) float xs[];          // [hidden]
    __shared__ float red[32];
    vm_pdl_launch_dependents();
    vm_pdl_wait();
    const int t = blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    stage_row<T>(x, norm_w, eps, t, hidden, xs, red);
    const int rows = top * ff + ff_shared;
    if (blockIdx.x == 0 && act_cols > rows)               // the input row, for the identity experts of the down kernel
        for (int i = threadIdx.x; i < hidden; i += blockDim.x) act[(size_t)t * act_cols + rows + i] = vm_from_float<T>(xs[i]);
    const int r0 = (blockIdx.x * nw + warp) * ROWS_PER_WARP;
    if (r0 >= rows) return;
    const W* wrow[ROWS_PER_WARP];
    const W* urow[ROWS_PER_WARP];
    int kind[ROWS_PER_WARP];
    bool routed[ROWS_PER_WARP], skip[ROWS_PER_WARP];
    float wgt[ROWS_PER_WARP];                             // glu == VM_GLU_SILU_WEIGHTED_INPUT: the routing weight scales the expert's input
    const int per = glu ? 2 * ff : ff;                    // rows of one expert's up matrix
#pragma unroll
    for (int i = 0; i < ROWS_PER_WARP; ++i) {
        const int r = min(r0 + i, rows - 1);              // (a row past the end repeats the last one and is not stored)
        routed[i] = r < top * ff;
        skip[i] = false;
        wgt[i] = 1.0f;
        if (routed[i]) {
            int e = chosen[(size_t)t * top + r / ff];
            if (glu == VM_GLU_SILU_WEIGHTED_INPUT) wgt[i] = weight[(size_t)t * top + r / ff];
            if (e >= E_real) { skip[i] = true; e = 0; }   // an identity expert has no rows: zeros
            wrow[i] = w_up + ((size_t)e * per + r % ff) * hidden;
            urow[i] = wrow[i] + (size_t)ff * hidden;
            kind[i] = act_kind;
        } else {
            wrow[i] = urow[i] = w_up_shared + (size_t)(r - top * ff) * hidden;
            if (glu >= VM_GLU_SILU_WEIGHTED_INPUT) urow[i] = wrow[i] + (size_t)ff_shared * hidden;      // the shared expert is gated too
            kind[i] = act_kind_shared;
        }
    }
    float d[ROWS_PER_WARP], u[ROWS_PER_WARP];
    warp_dot_rows<W, ROWS_PER_WARP>(wrow, xs, hidden, lane, d);
    if (glu) warp_dot_rows<W, ROWS_PER_WARP>(urow, xs, hidden, lane, u);
    if (lane == 0) {
#pragma unroll
        for (int i = 0; i < ROWS_PER_WARP; ++i)
            if (r0 + i < rows) {
                float v;
                if (skip[i]) v = 0.f;
                else if (glu >= VM_GLU_SILU_WEIGHTED_INPUT) {      // (VM_GLU_SILU: wgt stays 1, the weight is the down kernel's)
                    // W (w x) = w (W x): gate and up as the activation dtype holds them, the weight applied in float32
                    const float g = wgt[i] * vm_to_float(vm_from_float<T>(d[i])), uu = wgt[i] * vm_to_float(vm_from_float<T>(u[i]));
                    v = g / (1.0f + expf(-g)) * uu;
                } else if (glu && routed[i]) v = glu_clamped(vm_to_float(vm_from_float<T>(d[i])), vm_to_float(vm_from_float<T>(u[i])), limit, alpha);
                else v = expert_act(d[i], kind[i]);
                act[(size_t)t * act_cols + r0 + i] = vm_from_float<T>(v);
            }
    }
}

// ------------------------------------------------------------------------------------------------ down-projections
// grid (column tiles, T); a warp per output column
template <typename T, typename W>
__global__ void experts_down_kernel(const T* __restrict__ act, const W* __restrict__ w_down, const W* __restrict__ w_down_shared,
                                    const int* __restrict__ chosen, const float* __restrict__ weight, const float* __restrict__ shared_gate,
                                    int hidden, int ff, int ff_shared, int top, int E_real, int act_cols, int unit_weights, T* __restrict__ out,
                                    float* __restrict__ residual) {
    extern __shared__ __align__(16) float as[];          // [act_cols]: top * ff + ff_shared, then (identity experts) the input row
    vm_pdl_launch_dependents();
    vm_pdl_wait();
    const int t = blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int rows = top * ff + ff_shared;
    for (int i = threadIdx.x; i < act_cols; i += blockDim.x) as[i] = vm_to_float(act[(size_t)t * act_cols + i]);
    __syncthreads();
    const int c0 = (blockIdx.x * nw + warp) * ROWS_PER_WARP;
    if (c0 >= hidden) return;
    float y[ROWS_PER_WARP] = {};
    const W* wrow[ROWS_PER_WARP];
    float d[ROWS_PER_WARP];
    for (int k = 0; k < top; ++k) {
        const int e = chosen[(size_t)t * top + k];
        if (e >= E_real) {                                // an identity expert: the input itself, times the weight
            const float wk = weight[(size_t)t * top + k];
#pragma unroll
            for (int i = 0; i < ROWS_PER_WARP; ++i) y[i] = fmaf(wk, as[rows + min(c0 + i, hidden - 1)], y[i]);
            continue;
        }
#pragma unroll
        for (int i = 0; i < ROWS_PER_WARP; ++i) wrow[i] = w_down + ((size_t)e * hidden + min(c0 + i, hidden - 1)) * ff;
        warp_dot_rows<W, ROWS_PER_WARP>(wrow, as + k * ff, ff, lane, d);
        const float wk = unit_weights ? 1.0f : weight[(size_t)t * top + k];      // (the weight went into the expert's input)
#pragma unroll
        for (int i = 0; i < ROWS_PER_WARP; ++i) y[i] = fmaf(wk, d[i], y[i]);
    }
    if (ff_shared > 0) {
#pragma unroll
        for (int i = 0; i < ROWS_PER_WARP; ++i) wrow[i] = w_down_shared + (size_t)min(c0 + i, hidden - 1) * ff_shared;
        warp_dot_rows<W, ROWS_PER_WARP>(wrow, as + top * ff, ff_shared, lane, d);
        const float g = shared_gate ? shared_gate[t] : 1.0f;
#pragma unroll
        for (int i = 0; i < ROWS_PER_WARP; ++i) y[i] = fmaf(g, d[i], y[i]);
    }
    if (lane == 0) {
#pragma unroll
        for (int i = 0; i < ROWS_PER_WARP; ++i)
            if (c0 + i < hidden) {
                // into the float32 residual stream if one is given (through the activation dtype's rounding, as the unfused step adds it)
                if (residual) residual[(size_t)t * hidden + c0 + i] += vm_to_float(vm_from_float<T>(y[i]));
                else out[(size_t)t * hidden + c0 + i] = vm_from_float<T>(y[i]);
            }
    }
}

template <typename T, typename W>
int launch_experts(const void* x, const float* norm_w, float eps, const void* w_up, const void* w_down, const void* w_up_shared,
                   const void* w_down_shared, const int* chosen, const float* weight, const float* shared_gate, int T_, int hidden, int ff,
                   int ff_shared, int top, int act_kind, int act_kind_shared, int E_real, int n_identity, int glu, float limit, float alpha, void* act,
                   void* out, float* residual, cudaStream_t stream) {
    const int rows = top * ff + ff_shared;
    const int act_cols = rows + (n_identity > 0 ? hidden : 0);
    const int warps = 8;
    const size_t up_smem = (size_t)hidden * sizeof(float), down_smem = (size_t)act_cols * sizeof(float);
    if (up_smem > 200 * 1024 || down_smem > 200 * 1024) return VM_ERR_UNSUPPORTED;
    static VmOncePerDevice once[2];       // per instantiation
    if (up_smem > 48 * 1024 && vm_allow_smem(once[0], experts_up_kernel<T, W>, 200 * 1024) != cudaSuccess) return vm_launch_status();
    if (down_smem > 48 * 1024 && vm_allow_smem(once[1], experts_down_kernel<T, W>, 200 * 1024) != cudaSuccess) return vm_launch_status();
    const int per_block = warps * ROWS_PER_WARP;
    vm_launch_pdl(experts_up_kernel<T, W>, dim3((rows + per_block - 1) / per_block, T_), dim3(warps * 32), (size_t)hidden * sizeof(float), stream, x, norm_w, eps,
                  (const W*)w_up, (const W*)w_up_shared, chosen, hidden, ff, ff_shared, top, act_kind, act_kind_shared, E_real, glu, limit, alpha, act_cols,
                  weight, (T*)act);
    int st = vm_launch_status();
    if (st) return st;
    vm_launch_pdl(experts_down_kernel<T, W>, dim3((hidden + per_block - 1) / per_block, T_), dim3(warps * 32), down_smem, stream, (const T*)act,
                  (const W*)w_down, (const W*)w_down_shared, chosen, weight, shared_gate, hidden, ff, ff_shared, top, E_real, act_cols,
                  glu == VM_GLU_SILU_WEIGHTED_INPUT ? 1 : 0, (T*)out, residual);
    return vm_launch_status();
}

}  // namespace

// x, out [T, hidden] and the scratch `act` [T, vm_experts_act_cols(...)] in the activation dtype; expert weights stacked:
// w_up [E * ff, hidden] (glu: [E * 2 * ff, hidden], an expert's gate rows before its up rows), w_down [E * hidden, ff]; the shared expert's
// w_up_shared [ff_shared, hidden], w_down_shared [hidden, ff_shared] (ff_shared 0: none).  weight_dtype is the experts' storage.
// A chosen index >= E names an identity expert (n_identity of them): its result is the input row.  glu: act = glu_clamped(gate, up)
// with `limit` and `alpha`; else act_kind.
// norm_w given: x is the float32 residual stream, normed here.  residual given: the result is added into it and `out` is not written.
VM_API long long vm_experts_act_cols(int hidden, int ff, int ff_shared, int top, int n_identity) {
    return (long long)top * ff + ff_shared + (n_identity > 0 ? hidden : 0);
}

VM_API int vm_experts_few_tokens_glu(const void* x, const float* norm_w, float eps, const void* w_up, const void* w_down, const void* w_up_shared,
                                     const void* w_down_shared, int weight_dtype, const int* chosen, const float* weight, const float* shared_gate,
                                     int T, int hidden, int ff, int ff_shared, int top, int act_kind, int act_kind_shared, int E, int n_identity,
                                     int glu, float limit, float alpha, void* act, void* out, float* residual, int act_dtype, cudaStream_t stream) {
    if (T <= 0) return 0;
    if (hidden <= 0 || ff <= 0 || ff_shared < 0 || top <= 0 || E <= 0 || n_identity < 0) return VM_ERR_BAD_ARG;
    if (act_dtype == VM_F32 && weight_dtype == VM_F32)
        return launch_experts<float, float>(x, norm_w, eps, w_up, w_down, w_up_shared, w_down_shared, chosen, weight, shared_gate, T, hidden, ff, ff_shared,
                                            top, act_kind, act_kind_shared, E, n_identity, glu, limit, alpha, act, out, residual, stream);
    if (act_dtype == VM_BF16 && weight_dtype == VM_BF16)
        return launch_experts<__nv_bfloat16, __nv_bfloat16>(x, norm_w, eps, w_up, w_down, w_up_shared, w_down_shared, chosen, weight, shared_gate, T,
                                                            hidden, ff, ff_shared, top, act_kind, act_kind_shared, E, n_identity, glu, limit, alpha, act,
                                                            out, residual, stream);
    if (act_dtype == VM_BF16 && weight_dtype == VM_F32)
        return launch_experts<__nv_bfloat16, float>(x, norm_w, eps, w_up, w_down, w_up_shared, w_down_shared, chosen, weight, shared_gate, T, hidden, ff,
                                                    ff_shared, top, act_kind, act_kind_shared, E, n_identity, glu, limit, alpha, act, out, residual,
                                                    stream);
    return VM_ERR_UNSUPPORTED;
}

// the same for experts of one up matrix and an activation, every chosen index a real expert
VM_API int vm_experts_few_tokens(const void* x, const float* norm_w, float eps, const void* w_up, const void* w_down, const void* w_up_shared,
                                 const void* w_down_shared, int weight_dtype, const int* chosen, const float* weight, const float* shared_gate, int T,
                                 int hidden, int ff, int ff_shared, int top, int act_kind, int act_kind_shared, void* act, void* out,
                                 float* residual, int act_dtype, cudaStream_t stream) {
    return vm_experts_few_tokens_glu(x, norm_w, eps, w_up, w_down, w_up_shared, w_down_shared, weight_dtype, chosen, weight, shared_gate, T, hidden, ff,
                                     ff_shared, top, act_kind, act_kind_shared, 0x7fffffff, 0, 0, 0.f, 0.f, act, out, residual, act_dtype, stream);
}
