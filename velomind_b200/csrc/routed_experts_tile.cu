// The experts of few tokens in bfloat16 (decode steps): every expert streams its weight rows ONCE for all of its tokens, on mma.sync tiles.
// Arithmetic, arguments and layouts as in routed_experts.cu (products of bfloat16 with float32 sums, both gated forms, identity experts, a
// shared expert, the weighted sum in the order of a token's ranks).
//
// What bounds it is memory, the experts' weights: at 8 tokens of 4 experts each, 14 of 16 experts are in use (50 MB a layer at width 1,024, gated).
// Kernels that give every token its own pass over its experts read them 32 times (L2 carries 100 MB) and unpack every weight for one product:
// 23.5 us for the up-projections and 19.3 us for the down-projections of such a layer, 9.5 and 15.5 us for one token.  Here a block owns
// weight rows, finds the (token, expert) pairs that meet them, and multiplies rows with tokens on the tensor cores; a lane's 16-byte load of
// a weight row is the operand of two products (the contraction runs in the order the lanes hold it in).  Measured: 7.9 and 9.1 us, one token 4.1 and 5.4 us.
//   up:   a block per 16 rows of an expert (gated: 16 + 16), the contraction dealt out to its eight warps, joined in warp order.  With many pairs (as many
//         as experts, at least) the first weights are requested before the wait on the router: nearly every expert is met.
//   down: a block per 8 (or 16) output columns, for all experts: a warp takes an expert's rows 256 values of the contraction at a time,
//         the partial sums lie in shared memory by (pair, piece), and the last pass adds them up by rank and piece.
// No atomics, and nothing in a token's sums depends on the other tokens or on where its expert's list holds it.
#include <algorithm>

#include "mma.cuh"

namespace {

constexpr int UP_WARPS = 8;
constexpr int UP_KB = 4;                 // blocks of 32 of the contraction that a warp holds at a time
constexpr int UP_ROWS = 16;
constexpr int DOWN_WARPS = 16;
constexpr int DOWN_KB = 8;               // blocks of 32 of a piece
constexpr int DOWN_TOKENS = 32;          // tokens of a block
constexpr int MAX_PAIRS = 8192;          // (token, expert) pairs whose list an up block keeps in shared memory (32 KB behind 20 KB of sums: asked for below)

__device__ __forceinline__ float tile_act(float z, int kind) {
    if (kind == VM_ACT_RELU_SQUARED) { const float r = fmaxf(z, 0.f); return r * r; }
    if (kind == VM_ACT_GELU_TANH) return 0.5f * z * (1.0f + tanhf(0.7978845608028654f * (z + 0.044715f * z * z * z)));
    return z / (1.0f + expf(-z));
}
__device__ __forceinline__ float bf16_round(float v) { return __bfloat162float(__float2bfloat16_rn(v)); }
__device__ __forceinline__ uint4 zero4() { return make_uint4(0u, 0u, 0u, 0u); }

struct ExpertShape {
    int T, hidden, ff, ff_shared, top, E, n_identity, act_kind, act_kind_shared, glu, act_cols;
    float limit, alpha;
};

__device__ __forceinline__ float unit_value(const ExpertShape& z, float d, float u, float w, bool routed) {
    if (z.glu >= VM_GLU_SILU_WEIGHTED_INPUT) {             // W (w x) = w (W x): gate and up as bfloat16 holds them, the weight applied in float32
        const float g = w * bf16_round(d), uu = w * bf16_round(u);
        return g / (1.0f + expf(-g)) * uu;
    }
    if (z.glu && routed) {
        const float g = fminf(bf16_round(d), z.limit), uu = fminf(fmaxf(bf16_round(u), -z.limit), z.limit);
        return g / (1.0f + expf(-z.alpha * g)) * (uu + 1.0f);
    }
    return tile_act(d, routed ? z.act_kind : z.act_kind_shared);
}

// grid: E * ff / 16 blocks for the routed experts, then ff_shared / 16 for the shared one
__global__ void __launch_bounds__(UP_WARPS * 32, 2)
experts_up_tile_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ w_up, const __nv_bfloat16* __restrict__ w_up_shared,
                       const int* __restrict__ chosen, const float* __restrict__ weight, ExpertShape z, int eager, __nv_bfloat16* __restrict__ act) {
    extern __shared__ int list[];                          // the pairs (token * top + rank) of this block's expert
    __shared__ float part[UP_WARPS][2][UP_ROWS][10];       // [.., row, token]: 10 so that the lanes' pairs fall into different banks
    __shared__ int n_list;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t4 = lane & 3;
    const int tiles = z.ff / UP_ROWS, kbs = z.hidden / 32;
    const bool routed = (int)blockIdx.x < z.E * tiles;
    const int e = routed ? blockIdx.x / tiles : 0, r0 = (routed ? blockIdx.x - e * tiles : blockIdx.x - z.E * tiles) * UP_ROWS;
    const bool gated = routed ? z.glu != 0 : z.glu >= VM_GLU_SILU_WEIGHTED_INPUT;
    const int per = routed ? z.ff : z.ff_shared;           // rows of one of the expert's matrices; the up rows lie behind the gate rows
    const __nv_bfloat16* rows = (routed ? w_up + (size_t)e * (gated ? 2 : 1) * z.ff * z.hidden : w_up_shared) + (size_t)(r0 + g) * z.hidden + t4 * 8;
    const size_t to_up = (size_t)per * z.hidden;

    uint4 wa[2][UP_KB], wb[2][UP_KB];                      // rows g and g + 8 of the tile(s)
    auto load_weights = [&](int kb0) {
#pragma unroll
        for (int i = 0; i < UP_KB; ++i) {
            const bool ok = kb0 + i < kbs;
            const __nv_bfloat16* p = rows + (kb0 + i) * 32;
            wa[0][i] = ok ? *reinterpret_cast<const uint4*>(p) : zero4();
            wb[0][i] = ok ? *reinterpret_cast<const uint4*>(p + 8 * (size_t)z.hidden) : zero4();
            wa[1][i] = ok && gated ? *reinterpret_cast<const uint4*>(p + to_up) : zero4();
            wb[1][i] = ok && gated ? *reinterpret_cast<const uint4*>(p + to_up + 8 * (size_t)z.hidden) : zero4();
        }
    };
    const bool early = eager || !routed;
    if (early) load_weights(warp * UP_KB);                 // constants: nothing before this kernel writes them
    vm_pdl_launch_dependents();
    vm_pdl_wait();
    const int n_pairs = z.T * z.top;
    if (routed) {
        if (warp == 0) {
            int n = 0;
            for (int i0 = 0; i0 < n_pairs; i0 += 32) {
                const int i = i0 + lane;
                const bool mine = i < n_pairs && chosen[i] == e;
                const unsigned m = __ballot_sync(0xffffffffu, mine);
                if (mine) list[n + __popc(m & ((1u << lane) - 1u))] = i;
                n += __popc(m);
            }
            if (lane == 0) n_list = n;
        }
        __syncthreads();
    }
    const int n = routed ? n_list : z.T;
    if (n == 0) return;
    if (!early) load_weights(warp * UP_KB);
    const int step = UP_WARPS * UP_KB;
    for (int n0 = 0; n0 < n; n0 += 8) {
        const int p = n0 + g < n ? (routed ? list[n0 + g] : (n0 + g) * z.top) : -1;      // this lane's token, as a column of the product
        const __nv_bfloat16* xr = p >= 0 ? x + (size_t)(p / z.top) * z.hidden + t4 * 8 : nullptr;
        float c[2][4];
#pragma unroll
        for (int m = 0; m < 2; ++m) c[m][0] = c[m][1] = c[m][2] = c[m][3] = 0.f;
        for (int kb0 = warp * UP_KB; kb0 < kbs; kb0 += step) {
            uint4 b[UP_KB];
#pragma unroll
            for (int i = 0; i < UP_KB; ++i) b[i] = xr && kb0 + i < kbs ? *reinterpret_cast<const uint4*>(xr + (kb0 + i) * 32) : zero4();
            if (kb0 >= step || (n0 > 0 && kbs > step)) load_weights(kb0);
#pragma unroll
            for (int i = 0; i < UP_KB; ++i)
#pragma unroll
                for (int m = 0; m < 2; ++m) {
                    if (m == 1 && !gated) continue;
                    vm_mma_bf16_16816(c[m], wa[m][i].x, wb[m][i].x, wa[m][i].y, wb[m][i].y, b[i].x, b[i].y);
                    vm_mma_bf16_16816(c[m], wa[m][i].z, wb[m][i].z, wa[m][i].w, wb[m][i].w, b[i].z, b[i].w);
                }
        }
        if (n0 > 0) __syncthreads();                       // the sums of the tokens before are read
#pragma unroll
        for (int m = 0; m < 2; ++m) {
            *reinterpret_cast<float2*>(&part[warp][m][g][2 * t4]) = make_float2(c[m][0], c[m][1]);
            *reinterpret_cast<float2*>(&part[warp][m][g + 8][2 * t4]) = make_float2(c[m][2], c[m][3]);
        }
        __syncthreads();
        if (threadIdx.x < UP_ROWS * 8) {
            const int r = threadIdx.x & 15, col = threadIdx.x >> 4;
            if (n0 + col < n) {
                const int pair = routed ? list[n0 + col] : (n0 + col) * z.top, t = pair / z.top;
                float d = 0.f, u = 0.f;
#pragma unroll
                for (int w = 0; w < UP_WARPS; ++w) { d += part[w][0][r][col]; u += part[w][1][r][col]; }
                const float wgt = routed && z.glu == VM_GLU_SILU_WEIGHTED_INPUT ? weight[pair] : 1.0f;
                const int at = routed ? (pair - t * z.top) * z.ff + r0 + r : z.top * z.ff + r0 + r;
                act[(size_t)t * z.act_cols + at] = __float2bfloat16_rn(unit_value(z, d, u, wgt, routed));
            }
        }
    }
}

// grid (columns / (8 NT), token groups of DOWN_TOKENS)
template <int NT>
__global__ void __launch_bounds__(DOWN_WARPS * 32, 1)
experts_down_tile_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ act, const __nv_bfloat16* __restrict__ w_down,
                         const __nv_bfloat16* __restrict__ w_down_shared, const int* __restrict__ chosen, const float* __restrict__ weight,
                         const float* __restrict__ shared_gate, ExpertShape z, int piece, int unit_weights, __nv_bfloat16* __restrict__ out,
                         float* __restrict__ residual) {
    extern __shared__ __align__(16) float down_sm[];
    constexpr int COLS = 8 * NT;
    const int pieces = (z.ff + piece - 1) / piece, pieces_s = (z.ff_shared + piece - 1) / piece;
    float* part = down_sm;                                 // [DOWN_TOKENS * top][pieces][COLS], then the shared expert's [DOWN_TOKENS][pieces_s][COLS]
    float* part_s = part + (size_t)DOWN_TOKENS * z.top * pieces * COLS;
    int* pick = reinterpret_cast<int*>(part_s + (size_t)DOWN_TOKENS * pieces_s * COLS);      // [DOWN_TOKENS * top] the chosen outputs
    int* used = pick + DOWN_TOKENS * z.top;                // [E] whether an expert is met, then [E] the ones that are
    int* met = used + z.E;
    __shared__ int n_met;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t4 = lane & 3;
    const int t0 = blockIdx.y * DOWN_TOKENS, tokens = min(DOWN_TOKENS, z.T - t0), pairs = tokens * z.top;
    const int c0 = blockIdx.x * COLS;
    for (int i = threadIdx.x; i < z.E; i += blockDim.x) used[i] = 0;
    vm_pdl_launch_dependents();
    vm_pdl_wait();
    __syncthreads();
    for (int i = threadIdx.x; i < pairs; i += blockDim.x) {
        const int e = chosen[(size_t)t0 * z.top + i];
        pick[i] = e;
        if (e < z.E) used[e] = 1;
    }
    __syncthreads();
    if (warp == 0) {
        int n = 0;
        for (int e0 = 0; e0 < z.E; e0 += 32) {
            const bool hit = e0 + lane < z.E && used[e0 + lane];
            const unsigned m = __ballot_sync(0xffffffffu, hit);
            if (hit) met[n + __popc(m & ((1u << lane) - 1u))] = e0 + lane;
            n += __popc(m);
        }
        if (lane == 0) n_met = n;
    }
    __syncthreads();
    const int units = n_met * pieces + pieces_s;
    for (int u = warp; u < units; u += DOWN_WARPS) {
        const bool shared = u >= n_met * pieces;
        const int e = shared ? 0 : met[u / pieces], at = shared ? u - n_met * pieces : u % pieces;
        const int K = shared ? z.ff_shared : z.ff, k0 = at * piece, k1 = min(K, k0 + piece);
        const __nv_bfloat16* rows = (shared ? w_down_shared : w_down + (size_t)e * z.hidden * z.ff) + t4 * 8;
        // the tokens, sixteen at a time: for the shared expert all of them, else the pairs that chose e
        int from = 0, left = shared ? tokens : pairs;      // where to look on
        while (from < left) {
            int row[2] = {-1, -1};                         // rows g and g + 8 of the tile: a pair (shared: a token)
            int n = 0;
            if (shared) {
                n = min(16, left - from);
                if (g < n) row[0] = from + g;
                if (g + 8 < n) row[1] = from + g + 8;
                from += n;
            } else {
                while (from < left && n < 16) {
                    unsigned m = __ballot_sync(0xffffffffu, from + lane < left && pick[from + lane] == e);
                    const int have = __popc(m);
                    if (n + have > 16) {                   // the rest of this word's pairs belong to the next tile
                        for (int k = n + have - 16; k > 0; --k) m &= ~(0x80000000u >> __clz(m));
                    }
#pragma unroll
                    for (int half = 0; half < 2; ++half) {
                        const int k = g + 8 * half - n;
                        if (k >= 0 && k < __popc(m)) row[half] = from + (int)__fns(m, 0, k + 1);
                    }
                    n += __popc(m);
                    from += n == 16 ? 32 - __clz(m) : 32;
                }
                if (n == 0) break;
            }
            const __nv_bfloat16* ar[2];
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                const int t = shared ? row[half] : row[half] / z.top;
                ar[half] = row[half] < 0 ? nullptr
                                         : act + (size_t)(t0 + t) * z.act_cols + (shared ? z.top * z.ff : (row[half] - t * z.top) * z.ff) + t4 * 8;
            }
            float c[NT][4];
#pragma unroll
            for (int i = 0; i < NT; ++i) c[i][0] = c[i][1] = c[i][2] = c[i][3] = 0.f;
            for (int k = k0; k < k1; k += DOWN_KB * 32) {
                uint4 wv[NT][DOWN_KB], a[2][DOWN_KB];
#pragma unroll
                for (int i = 0; i < NT; ++i)
#pragma unroll
                    for (int kb = 0; kb < DOWN_KB; ++kb)
                        wv[i][kb] = k + kb * 32 < k1 ? *reinterpret_cast<const uint4*>(rows + (size_t)(c0 + i * 8 + g) * K + k + kb * 32) : zero4();
#pragma unroll
                for (int half = 0; half < 2; ++half)
#pragma unroll
                    for (int kb = 0; kb < DOWN_KB; ++kb)
                        a[half][kb] = ar[half] && k + kb * 32 < k1 ? *reinterpret_cast<const uint4*>(ar[half] + k + kb * 32) : zero4();
#pragma unroll
                for (int kb = 0; kb < DOWN_KB; ++kb)
#pragma unroll
                    for (int i = 0; i < NT; ++i) {
                        vm_mma_bf16_16816(c[i], a[0][kb].x, a[1][kb].x, a[0][kb].y, a[1][kb].y, wv[i][kb].x, wv[i][kb].y);
                        vm_mma_bf16_16816(c[i], a[0][kb].z, a[1][kb].z, a[0][kb].w, a[1][kb].w, wv[i][kb].z, wv[i][kb].w);
                    }
            }
            float* base = shared ? part_s : part;
            const int n_pieces = shared ? pieces_s : pieces;
#pragma unroll
            for (int half = 0; half < 2; ++half)
                if (row[half] >= 0)
#pragma unroll
                    for (int i = 0; i < NT; ++i)
                        *reinterpret_cast<float2*>(base + ((size_t)row[half] * n_pieces + at) * COLS + i * 8 + 2 * t4) = make_float2(c[i][2 * half], c[i][2 * half + 1]);
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < tokens * COLS; i += blockDim.x) {
        const int t = i / COLS, col = i - t * COLS;
        float y = 0.f;
        for (int k = 0; k < z.top; ++k) {
            const int e = pick[t * z.top + k];
            const float w = weight[(size_t)t0 * z.top + t * z.top + k];
            if (e >= z.E) {                                // an identity expert: the input itself, times the weight
                y = fmaf(w, __bfloat162float(x[(size_t)(t0 + t) * z.hidden + c0 + col]), y);
                continue;
            }
            float d = 0.f;
            for (int s = 0; s < pieces; ++s) d += part[((size_t)(t * z.top + k) * pieces + s) * COLS + col];
            y = fmaf(unit_weights ? 1.0f : w, d, y);       // (the weight went into the expert's input)
        }
        if (pieces_s > 0) {
            float d = 0.f;
            for (int s = 0; s < pieces_s; ++s) d += part_s[((size_t)t * pieces_s + s) * COLS + col];
            y = fmaf(shared_gate ? shared_gate[t0 + t] : 1.0f, d, y);
        }
        const size_t o = (size_t)(t0 + t) * z.hidden + c0 + col;
        // into the float32 residual stream if one is given (through bfloat16's rounding, as the unfused step adds it)
        if (residual) residual[o] += bf16_round(y);
        else out[o] = __float2bfloat16_rn(y);
    }
}

// values of the contraction in one piece of the down kernel: 256, or so many that there are at most eight pieces (a function of the expert's size alone)
int down_piece(int ff, int ff_shared) {
    int p = DOWN_KB * 32;
    while (8 * p < std::max(ff, ff_shared)) p *= 2;
    return p;
}
size_t down_smem(int ff, int ff_shared, int top, int E, int nt) {
    const int p = down_piece(ff, ff_shared);
    return ((size_t)DOWN_TOKENS * top * ((ff + p - 1) / p) + (size_t)DOWN_TOKENS * ((ff_shared + p - 1) / p)) * 8 * nt * sizeof(float) +
           ((size_t)DOWN_TOKENS * top + 2 * (size_t)E) * sizeof(int);
}
int down_tiles(int hidden) { return hidden % 16 == 0 && hidden / 8 > vm_sm_count() ? 2 : 1; }      // 16 columns a block once 8 would make more blocks than SMs

bool aligned16(const void* p) { return reinterpret_cast<uintptr_t>(p) % 16 == 0; }

}  // namespace

// 1 if vm_experts_few_tile takes these sizes (rows of whole 16-byte pieces in blocks of 32, lists and partial sums that fit shared memory)
VM_API int vm_experts_few_tile_fits(int T, int hidden, int ff, int ff_shared, int top, int E, int n_identity) {
    if (T <= 0 || hidden <= 0 || ff <= 0 || ff_shared < 0 || top <= 0 || E <= 0 || n_identity < 0) return 0;
    if (hidden % 32 || ff % 32 || ff_shared % 32 || (long long)T * top > MAX_PAIRS || E > 1024 || top > 64) return 0;
    if (vm_experts_act_cols(hidden, ff, ff_shared, top, n_identity) % 8) return 0;
    return down_smem(ff, ff_shared, top, E, 2) <= 200 * 1024 ? 1 : 0;
}

// x [T, hidden] bfloat16 rows (normed); weights, act and out bfloat16; the other arguments as vm_experts_few_tokens_glu (the input row behind act's
// columns is not written: the down kernel reads x).  T rows of everything.
VM_API int vm_experts_few_tile(const void* x, const void* w_up, const void* w_down, const void* w_up_shared, const void* w_down_shared, const int* chosen,
                               const float* weight, const float* shared_gate, int T, int hidden, int ff, int ff_shared, int top, int act_kind,
                               int act_kind_shared, int E, int n_identity, int glu, float limit, float alpha, void* act, void* out, float* residual,
                               cudaStream_t stream) {
    if (T <= 0) return 0;
    if (!vm_experts_few_tile_fits(T, hidden, ff, ff_shared, top, E, n_identity)) return VM_ERR_UNSUPPORTED;
    if (!aligned16(x) || !aligned16(w_up) || !aligned16(w_down) || !aligned16(w_up_shared) || !aligned16(w_down_shared) || !aligned16(act)) return VM_ERR_UNSUPPORTED;
    const ExpertShape z{T, hidden, ff, ff_shared, top, E, n_identity, act_kind, act_kind_shared, glu,
                        (int)vm_experts_act_cols(hidden, ff, ff_shared, top, n_identity), limit, alpha};
    const int nt = down_tiles(hidden);
    const size_t smem = down_smem(ff, ff_shared, top, E, nt);
    static VmOncePerDevice once[3];
    cudaError_t e = vm_allow_smem(once[0], experts_up_tile_kernel, MAX_PAIRS * sizeof(int));
    if (e == cudaSuccess) e = nt == 2 ? vm_allow_smem(once[2], experts_down_tile_kernel<2>, 200 * 1024) : vm_allow_smem(once[1], experts_down_tile_kernel<1>, 200 * 1024);
    if (e != cudaSuccess) return (int)e;
    vm_launch_pdl(experts_up_tile_kernel, dim3(E * (ff / UP_ROWS) + ff_shared / UP_ROWS), dim3(UP_WARPS * 32), (size_t)T * top * sizeof(int), stream,
                  (const __nv_bfloat16*)x, (const __nv_bfloat16*)w_up, (const __nv_bfloat16*)w_up_shared, chosen, weight, z, T * top >= E ? 1 : 0,
                  (__nv_bfloat16*)act);
    const int st = vm_launch_status();
    if (st) return st;
    vm_launch_pdl(nt == 2 ? experts_down_tile_kernel<2> : experts_down_tile_kernel<1>, dim3(hidden / (8 * nt), (T + DOWN_TOKENS - 1) / DOWN_TOKENS),
                  dim3(DOWN_WARPS * 32), smem, stream, (const __nv_bfloat16*)x, (const __nv_bfloat16*)act, (const __nv_bfloat16*)w_down,
                  (const __nv_bfloat16*)w_down_shared, chosen, weight, shared_gate, z, down_piece(ff, ff_shared), glu == VM_GLU_SILU_WEIGHTED_INPUT ? 1 : 0,
                  (__nv_bfloat16*)out, residual);
    return vm_launch_status();
}
