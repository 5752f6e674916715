// out[T, N] = x[T, K] W[N, K]^T in float32 for up to eight rows of x: the products of a decode step in the true 32-bit path, with the norm in front,
// the residual sum behind or the gated unit fused in where the part asks for it (a norm of its own took 4.2 us, a unit 2.3 us).
//
// What bounds it is the weights' way through memory, and at these sizes the latency of it (1.3 MB for N = K = 576).  The library's kernels for a
// few rows took 9.4 us (4 rows; a block walks a weight row with a chain of loads) to 14 us (two launches, the sum split).  Here a block owns four
// weight rows and its warps share the contraction: every load of a block is in flight at once, a float4 per lane and row, requested before the
// wait on the kernel in front (weights are constants); x comes from L2 a float4 per row.  The 4 x rows sums of a warp are reduced together, each
// shuffle halving what a lane still holds, and the warps' sums meet in shared memory in warp order.  Measured in a decode step of 4 rows: 960 x 576 with
// the norm 2.7 us, 3,072 x 576 with the norm and the unit 5.5 us, 576 x 576 and 576 x 1,536 with the residual sum 3.2 us, 49,152 x 576 35 us (113 MB).
// A row's result does not depend on the other rows of x.
#include "common.cuh"

namespace {

constexpr int RN = 4;                    // weight rows of a block
constexpr int MAX_WARPS = 8;

// v[0 .. V) of every lane summed over the warp; afterwards lane i holds the total of value i / (32 / V) in v[0]
template <int V> __device__ __forceinline__ void reduce_together(float (&v)[V], int lane) {
    int o = 16;
#pragma unroll
    for (int n = V / 2; n >= 1; n /= 2, o /= 2) {          // a lane passes on the half that its partner keeps
        const bool up = lane & o;
#pragma unroll
        for (int i = 0; i < n; ++i) {
            const float give = up ? v[i] : v[i + n], keep = up ? v[i + n] : v[i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
        }
    }
#pragma unroll
    for (; o >= 1; o /= 2) v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
}

enum { F32_STORE = 0, F32_RESIDUAL = 1, F32_SWIGLU = 2 };

// NORM: the rows of x are normed on the way, out = (x norm_w / rms(x)) W^T: the weights of the norm go into the products, the sum of squares is
// taken beside them and divides the result.  MODE: store; add into out; W = [gate; up] stacked, out[T, N / 2] = silu(gate) up (a block owns two
// rows of either half).
template <int M, bool NORM, int MODE>
__global__ void __launch_bounds__(MAX_WARPS * 32)
skinny_f32_kernel(const float* __restrict__ x, long long ldx, const float* __restrict__ norm_w, float eps, const float* __restrict__ w, float* __restrict__ out,
                  int T, int N, int K) {
    constexpr int V = RN * M;
    __shared__ float part[MAX_WARPS][V], squares[MAX_WARPS][M];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, step = blockDim.x * 4, warps = blockDim.x / 32;
    const int n0 = blockIdx.x * (MODE == F32_SWIGLU ? RN / 2 : RN), cols = MODE == F32_SWIGLU ? N / 2 : N;
    auto row = [&](int r) { return MODE == F32_SWIGLU ? (r < RN / 2 ? n0 + r : cols + n0 + r - RN / 2) : n0 + r; };
    auto there = [&](int r) { return n0 + (MODE == F32_SWIGLU ? r % (RN / 2) : r) < cols; };
    float4 wv[RN], nv = make_float4(1.f, 1.f, 1.f, 1.f);
    auto load = [&](int k) {
#pragma unroll
        for (int r = 0; r < RN; ++r)
            wv[r] = k < K && there(r) ? __ldcs(reinterpret_cast<const float4*>(w + (size_t)row(r) * K + k)) : make_float4(0.f, 0.f, 0.f, 0.f);
        if (NORM && k < K) nv = *reinterpret_cast<const float4*>(norm_w + k);
    };
    int k = threadIdx.x * 4;
    load(k);
    vm_pdl_launch_dependents();
    vm_pdl_wait();
    float v[V], ss[M];
#pragma unroll
    for (int i = 0; i < V; ++i) v[i] = 0.f;
#pragma unroll
    for (int m = 0; m < M; ++m) ss[m] = 0.f;
    for (; k < K; k += step) {
        float4 xv[M];
#pragma unroll
        for (int m = 0; m < M; ++m) xv[m] = m < T ? *reinterpret_cast<const float4*>(x + (size_t)m * ldx + k) : make_float4(0.f, 0.f, 0.f, 0.f);
        if (NORM) {
#pragma unroll
            for (int m = 0; m < M; ++m) {
                ss[m] = fmaf(xv[m].x, xv[m].x, fmaf(xv[m].y, xv[m].y, fmaf(xv[m].z, xv[m].z, fmaf(xv[m].w, xv[m].w, ss[m]))));
                xv[m].x *= nv.x; xv[m].y *= nv.y; xv[m].z *= nv.z; xv[m].w *= nv.w;
            }
        }
#pragma unroll
        for (int r = 0; r < RN; ++r)
#pragma unroll
            for (int m = 0; m < M; ++m) {
                float& a = v[r * M + m];
                a = fmaf(wv[r].x, xv[m].x, a); a = fmaf(wv[r].y, xv[m].y, a);
                a = fmaf(wv[r].z, xv[m].z, a); a = fmaf(wv[r].w, xv[m].w, a);
            }
        load(k + step);
    }
    reduce_together<V>(v, lane);
    if (lane % (32 / V) == 0) part[warp][lane / (32 / V)] = v[0];
    if (NORM) {
        reduce_together<M>(ss, lane);
        if (lane % (32 / M) == 0) squares[warp][lane / (32 / M)] = ss[0];
    }
    __syncthreads();
    const int r = threadIdx.x / M, m = threadIdx.x % M;
    if (threadIdx.x >= (MODE == F32_SWIGLU ? V / 2 : V) || m >= T || !there(r)) return;
    float inv = 1.0f;
    if (NORM) {
        float sum = 0.f;
        for (int i = 0; i < warps; ++i) sum += squares[i][m];
        inv = 1.0f / sqrtf(sum / (float)K + eps);
    }
    float sum = 0.f;
    for (int i = 0; i < warps; ++i) sum += part[i][threadIdx.x];
    sum *= inv;
    float* o = out + (size_t)m * cols + n0 + r;
    if (MODE == F32_SWIGLU) {
        float up = 0.f;
        for (int i = 0; i < warps; ++i) up += part[i][threadIdx.x + V / 2];
        up *= inv;
        *o = sum / (1.0f + expf(-sum)) * up;
    } else if (MODE == F32_RESIDUAL) {
        *o += sum;
    } else {
        *o = sum;
    }
}

template <bool NORM, int MODE>
int launch_f32(const float* x, long long ldx, const float* norm_w, float eps, const float* w, float* out, int T, int N, int K, cudaStream_t stream) {
    const int warps = (K + 127) / 128 < MAX_WARPS ? (K + 127) / 128 : MAX_WARPS;      // a float4 per lane, row and turn
    const dim3 grid((N + RN - 1) / RN), block(warps * 32);
    if (T == 1) vm_launch_pdl(skinny_f32_kernel<1, NORM, MODE>, grid, block, 0, stream, x, ldx, norm_w, eps, w, out, T, N, K);
    else if (T == 2) vm_launch_pdl(skinny_f32_kernel<2, NORM, MODE>, grid, block, 0, stream, x, ldx, norm_w, eps, w, out, T, N, K);
    else if (T <= 4) vm_launch_pdl(skinny_f32_kernel<4, NORM, MODE>, grid, block, 0, stream, x, ldx, norm_w, eps, w, out, T, N, K);
    else vm_launch_pdl(skinny_f32_kernel<8, NORM, MODE>, grid, block, 0, stream, x, ldx, norm_w, eps, w, out, T, N, K);
    return vm_launch_status();
}

}  // namespace

// 1 if vm_skinny_f32 takes these rows (at most eight, whole 16-byte pieces)
VM_API int vm_skinny_f32_fits(const void* x, long long ldx, const void* w, int T, int K) {
    return T >= 1 && T <= 8 && K % 4 == 0 && ldx % 4 == 0 && reinterpret_cast<uintptr_t>(x) % 16 == 0 && reinterpret_cast<uintptr_t>(w) % 16 == 0 ? 1 : 0;
}

// x float32 [T, K] with rows ldx apart, w float32 [N, K], out float32 [T, N]
VM_API int vm_skinny_f32(const float* x, long long ldx, const float* w, float* out, int T, int N, int K, cudaStream_t stream) {
    return vm_skinny_f32_fused(x, ldx, nullptr, 0.f, w, out, T, N, K, 0, 0, stream);
}

// the same with the neighbouring work: norm_w [K] given, the rows of x are normed (out = rmsnorm(x) W^T); add: out += instead of out =; swiglu (with
// norm_w or without): w = [gate; up] stacked (N rows together), out [T, N / 2] = silu(x gate^T) (x up^T)
VM_API int vm_skinny_f32_fused(const float* x, long long ldx, const float* norm_w, float eps, const float* w, float* out, int T, int N, int K, int add,
                               int swiglu, cudaStream_t stream) {
    if (T <= 0 || N <= 0) return 0;
    if (K <= 0 || (add && swiglu) || (swiglu && N % 2) || !vm_skinny_f32_fits(x, ldx, w, T, K) || reinterpret_cast<uintptr_t>(norm_w) % 16) return VM_ERR_UNSUPPORTED;
    if (norm_w) {
        if (swiglu) return launch_f32<true, F32_SWIGLU>(x, ldx, norm_w, eps, w, out, T, N, K, stream);
        if (add) return launch_f32<true, F32_RESIDUAL>(x, ldx, norm_w, eps, w, out, T, N, K, stream);
        return launch_f32<true, F32_STORE>(x, ldx, norm_w, eps, w, out, T, N, K, stream);
    }
    if (swiglu) return launch_f32<false, F32_SWIGLU>(x, ldx, norm_w, eps, w, out, T, N, K, stream);
    if (add) return launch_f32<false, F32_RESIDUAL>(x, ldx, norm_w, eps, w, out, T, N, K, stream);
    return launch_f32<false, F32_STORE>(x, ldx, norm_w, eps, w, out, T, N, K, stream);
}
