// out[T, N] = x[T, K] W[N, K]^T in float32 for many rows (prompts of the true 32-bit path) on the fifth-generation tensor cores.
//
// A float32 value is the sum of three bfloat16 values to the last bit or nearly so (24 bits of mantissa, 8 + 8 + 8 with signs of their own), and a product
// of two bfloat16 values is exact in float32.  So x w = xh wh + (xh wm + xm wh + xm wm + xh wl + xl wh) with what is left out below 2^-25 of |x w|.  The
// tensor cores' own float32 sums are cut off, not rounded, so the large products (xh wh) stay in tensor memory for 64 places of K only and are then added to
// float32 registers with rounding; the small ones (2^-8 of the sum) keep an accumulator of their own for all of K.
//
// What bounds it is the hand-over of a step of 64 places from the splitting warps to the tensor cores and back (1.2 us at the fewest rows), then the splitting, eight
// instructions a value, not the six products: a CTA takes 128 rows by 32 or 64 columns, whichever keeps the waves over the SMs and the values split per CTA low
// (choose_columns).  Warps 0..7 split the values of 64 places of K into the shared-memory tiles (K-major, 128-byte rows, 128-byte swizzle; two stages) with the
// values of the next two steps on their way into registers; they are asked for behind the proxy fence of a step, which waits for loads in flight.  Warp 12
// issues the products (tcgen05.mma, M = 128, K = 16), warps 8..11 empty the accumulator of the large products, which lies twice in tensor memory.
//
// Measured against the library's float32 product: 446 rows, 3,072 x 576 32 / 43.7 us, 960 x 576 15.2 / 17.6, 1,024 x 2,816 57 / 72, 5,632 x 1,024 74 / 118; 130 rows,
// 4,128 x 1,024 27.4 / 46.8; 1,000 rows, 5,632 x 1,024 127 / 247; 33 rows, 5,632 x 1,024 24.3 / 31.5.  Below some 350,000 cells it is no faster: 446 rows, 576 x 576
// 14.6 / 13.3, 576 x 1,536 32.3 / 30.2; 130 rows, 960 x 576 14.3 / 12.7.  Nor is it up to 32 rows, for which the library has kernels of its own, however many the
// columns: 9 rows, 49,152 x 576 79 / 50, 49,152 x 2,048 236 / 158; 32 rows 83 / 51, 244 / 163, 12,288 x 2,048 112 / 68; but 33 rows 86 / 83, 252 / 311, 85 / 86;
// 64 rows 90 / 97, 259 / 321, 88 / 86, 32,000 x 1,024 95 / 87; 96 rows and more are faster at every size.  2-norm of the error against 64 bits, of the result's: 0.9 to 1.5 x 10^-7 / 4 to 9 x 10^-7.
//
// What the parts cannot express is computed again, cell by cell, with fused multiply-adds straight from memory, as all cells are after a wait that ran out: the
// cells of a row or column with a value that bfloat16 cannot hold (infinities, NaN, above its largest finite value); cells whose sum is not finite (of operands
// whose product passes float32's range the large sum holds an infinity and a small one, whose parts have signs of their own, may hold the other); and cells so
// small beside their row and column that low parts below the smallest normal number, which the tensor cores may take for zero, could show in the last place
// (pf_smallest).  Looking costs 0.2 to 0.5 us a CTA; one infinity in 446 rows, 3,072 x 576 32 -> 56 us.
//
// Sizes: K % 4 == 0, 16-byte rows.  A row's result does not depend on the other rows: which way a cell goes depends on its row, its column and its sum alone.
#include "tc05.cuh"

namespace {

constexpr int PF_ROWS = 128, PF_K = 64, PF_SPLITTERS = 8, PF_DRAINERS = 4, PF_STAGES = 2;
constexpr int PF_THREADS = (PF_SPLITTERS + PF_DRAINERS + 1) * 32;
constexpr float PF_LARGEST = 3.38e38f;                   // below what rounds to infinity in bfloat16 (3.3953e38)

__device__ __forceinline__ float pf_max_nan(float a, float b) {      // NaN if either is
    float y;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(y) : "f"(a), "f"(b));
    return y;
}

// Below this a sum may have lost something that matters.  Parts, products and sums below 2^-126 may be taken for zero: at most three parts of a value times the other
// operand (at most `most_x` and `most_w`), and six products, at each of K places; that is 2^-24 of the sum and less from here on.
__device__ __forceinline__ float pf_smallest(int K, float most_x, float most_w) { return (float)K * 1.9721523e-31f * (6.f + 3.f * (most_x + most_w)); }      // (2^-102)

__device__ __forceinline__ void pf_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]),
                   "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(taddr) : "memory");
}

// two values into their three parts, packed
__device__ __forceinline__ void pf_split(float a, float b, uint32_t& h, uint32_t& m, uint32_t& l) {
    h = vm_pack_bf16(a, b);
    a -= __uint_as_float(h << 16); b -= __uint_as_float(h & 0xffff0000u);
    m = vm_pack_bf16(a, b);
    a -= __uint_as_float(m << 16); b -= __uint_as_float(m & 0xffff0000u);
    l = vm_pack_bf16(a, b);
}

template <int BN>
__global__ void __launch_bounds__(PF_THREADS, 1)
products_f32_kernel(const float* __restrict__ x, long long ldx, const float* __restrict__ W, float* __restrict__ out, int T, int N, int K) {
    constexpr uint32_t A_PART = PF_ROWS * PF_K * 2, B_PART = BN * PF_K * 2, STAGE = 3 * (A_PART + B_PART);
    constexpr uint32_t COLS = 3 * BN <= 128 ? 128 : 256;      // two accumulators of the large products, one of the small ones
    // float32 sums (bits 4-5 = 1), A and B bfloat16 (bits 7-9, 10-12 = 1), both K-major, N >> 3 in bits 17-22, M >> 4 in bits 24-28
    constexpr uint32_t IDESC = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(PF_ROWS >> 4) << 24);
    constexpr int AJ = PF_ROWS / 32, PIECES = AJ + BN / 32;      // pieces of eight values that a splitting thread takes: eighth tid % 8 of rows tid / 8 + 32 j of x, then of W
    extern __shared__ __align__(1024) unsigned char tiles[];
    __shared__ __align__(8) unsigned long long bars[9];  // full[2], empty[2], large full[2], large free[2], done
    __shared__ uint32_t tmem_slot;
    __shared__ int gave_up;
    __shared__ float most[PF_ROWS + BN];                 // the largest magnitude of each row of x, of each row of W
    __shared__ uint32_t again[PF_ROWS][BN / 32];         // cells to be computed again
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int m0 = blockIdx.y * PF_ROWS, n0 = blockIdx.x * BN, steps = (K + PF_K - 1) / PF_K;
    const uint32_t full0 = ta_u32(&bars[0]), empty0 = ta_u32(&bars[2]), large0 = ta_u32(&bars[4]), free0 = ta_u32(&bars[6]), done = ta_u32(&bars[8]);
    if (tid == 0) {
        gave_up = (ta_u32(tiles) & 1023u) ? 1 : 0;       // (misaligned tiles would give wrong sums)
        for (int s = 0; s < 2; ++s) {
            ta_bar_init(full0 + 8 * s, PF_SPLITTERS); ta_bar_init(empty0 + 8 * s, 1);
            ta_bar_init(large0 + 8 * s, 1); ta_bar_init(free0 + 8 * s, PF_DRAINERS);
        }
        ta_bar_init(done, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == PF_SPLITTERS + PF_DRAINERS) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(ta_u32(&tmem_slot)), "r"(COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    ta_fence_before();
    __syncthreads();
    ta_fence_after();
    const uint32_t tmem = tmem_slot;
    volatile int* abort_p = &gave_up;
    vm_pdl_wait();
    vm_pdl_launch_dependents();

    float sums[BN];                                      // of a draining thread: row m0 + 32 (warp % 4) + lane
#pragma unroll
    for (int j = 0; j < BN; ++j) sums[j] = 0.f;
    const int quarter = warp & 3;
    if (warp < PF_SPLITTERS) {
        const int eighth = tid & 7, r0 = tid >> 3;
        const float* xa = x + (size_t)(m0 + r0) * ldx + eighth * 8;
        const float* wb = W + (size_t)(n0 + r0) * K + eighth * 8;
        // (rows past the last are neither split nor cleared: what their tiles hold enters cells that are not stored)
        auto there = [&](int j) { return j < AJ ? m0 + r0 + 32 * j < T : n0 + r0 + 32 * (j - AJ) < N; };
        float largest[PIECES];
#pragma unroll
        for (int j = 0; j < PIECES; ++j) largest[j] = 0.f;
        auto fetch = [&](float4 (&v)[PIECES][2], int step) {
            const int k = step * PF_K + eighth * 8;
#pragma unroll
            for (int j = 0; j < PIECES; ++j) {
                const float4* at = reinterpret_cast<const float4*>((j < AJ ? xa + (size_t)(32 * j) * ldx : wb + (size_t)(32 * (j - AJ)) * K) + step * PF_K);
                v[j][0] = v[j][1] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (there(j) && k < K) v[j][0] = __ldg(at);
                if (there(j) && k + 4 < K) v[j][1] = __ldg(at + 1);
            }
        };
        auto put = [&](const float4 (&v)[PIECES][2], int i) {
            const int s = i & 1;
            if (!ta_spin(empty0 + 8 * s, ((uint32_t)(i >> 1) & 1u) ^ 1u, abort_p)) return false;
#pragma unroll
            for (int j = 0; j < PIECES; ++j) {
                if (!there(j)) continue;
                const uint32_t part = j < AJ ? A_PART : B_PART;
                const int row = j < AJ ? r0 + 32 * j : r0 + 32 * (j - AJ);
                uint4 h, m, l;
                pf_split(v[j][0].x, v[j][0].y, h.x, m.x, l.x); pf_split(v[j][0].z, v[j][0].w, h.y, m.y, l.y);
                pf_split(v[j][1].x, v[j][1].y, h.z, m.z, l.z); pf_split(v[j][1].z, v[j][1].w, h.w, m.w, l.w);
                largest[j] = pf_max_nan(pf_max_nan(pf_max_nan(fabsf(v[j][0].x), fabsf(v[j][0].y)), pf_max_nan(fabsf(v[j][0].z), fabsf(v[j][0].w))), largest[j]);
                largest[j] = pf_max_nan(pf_max_nan(pf_max_nan(fabsf(v[j][1].x), fabsf(v[j][1].y)), pf_max_nan(fabsf(v[j][1].z), fabsf(v[j][1].w))), largest[j]);
                unsigned char* at = tiles + s * STAGE + (j < AJ ? 0u : 3 * A_PART) + row * 128 + ((eighth ^ (row & 7)) << 4);
                *reinterpret_cast<uint4*>(at) = h;
                *reinterpret_cast<uint4*>(at + part) = m;
                *reinterpret_cast<uint4*>(at + 2 * part) = l;
            }
            ta_fence_async_smem();
            __syncwarp();
            if (lane == 0) ta_bar_arrive(full0 + 8 * s);
            return true;
        };
        float4 even[PIECES][2], odd[PIECES][2];
        fetch(even, 0);
        fetch(odd, 1);
        for (int i = 0; i < steps; i += 2) {
            if (!put(even, i)) break;
            fetch(even, i + 2);
            if (i + 1 >= steps || !put(odd, i + 1)) break;
            fetch(odd, i + 3);
        }
#pragma unroll
        for (int j = 0; j < PIECES; ++j) {               // (eight neighbouring lanes have a row)
#pragma unroll
            for (int o = 1; o < 8; o *= 2) largest[j] = pf_max_nan(largest[j], __shfl_xor_sync(0xffffffffu, largest[j], o));
            if (eighth == 0) most[j < AJ ? r0 + 32 * j : PF_ROWS + r0 + 32 * (j - AJ)] = largest[j];
        }
    } else if (warp == PF_SPLITTERS + PF_DRAINERS) {
        if (lane == 0) {
            for (int i = 0; i < steps; ++i) {
                const int s = i & 1;
                if (!ta_spin(free0 + 8 * s, ((uint32_t)(i >> 1) & 1u) ^ 1u, abort_p)) break;
                if (!ta_spin(full0 + 8 * s, (uint32_t)(i >> 1) & 1u, abort_p)) break;
                ta_fence_after();
                const uint32_t at = ta_u32(tiles) + s * STAGE;
                uint64_t da[3], db[3];
#pragma unroll
                for (int part = 0; part < 3; ++part) { da[part] = ta_desc(at + part * A_PART); db[part] = ta_desc(at + 3 * A_PART + part * B_PART); }
                const uint32_t large = tmem + (uint32_t)(s * BN), small = tmem + 2u * BN;
#pragma unroll
                for (int k = 0; k < PF_K / 16; ++k) ta_mma(large, da[0] + 2 * k, db[0] + 2 * k, IDESC, k > 0 ? 1u : 0u);
                ta_commit(large0 + 8 * s);
#pragma unroll
                for (int k = 0; k < PF_K / 16; ++k) {
                    ta_mma(small, da[0] + 2 * k, db[2] + 2 * k, IDESC, i > 0 || k > 0 ? 1u : 0u);
                    ta_mma(small, da[2] + 2 * k, db[0] + 2 * k, IDESC, 1u);
                    ta_mma(small, da[1] + 2 * k, db[1] + 2 * k, IDESC, 1u);
                    ta_mma(small, da[0] + 2 * k, db[1] + 2 * k, IDESC, 1u);
                    ta_mma(small, da[1] + 2 * k, db[0] + 2 * k, IDESC, 1u);
                }
                ta_commit(empty0 + 8 * s);
            }
            ta_commit(done);                             // (of all products issued, after a wait that ran out too)
        }
        __syncwarp();
    } else {
        const uint32_t mine = tmem + ((uint32_t)(quarter * 32) << 16);
        auto add = [&](uint32_t at) {
#pragma unroll
            for (int p = 0; p < BN; p += 16) {
                uint32_t v[16];
                pf_ld16(at + p, v);
                ta_ld_wait();
#pragma unroll
                for (int j = 0; j < 16; ++j) sums[p + j] += __uint_as_float(v[j]);
            }
        };
        bool ok = true;
        for (int i = 0; i < steps; ++i) {
            const int s = i & 1;
            ok = __all_sync(0xffffffffu, ta_spin(large0 + 8 * s, (uint32_t)(i >> 1) & 1u, abort_p));
            if (!ok) break;
            ta_fence_after();
            add(mine + (uint32_t)(s * BN));
            ta_fence_before();
            __syncwarp();
            if (lane == 0) ta_bar_arrive(free0 + 8 * s);
        }
        ok = __all_sync(0xffffffffu, ta_spin(done, 0u, abort_p)) && ok;      // (the tensor memory goes back once nothing writes it)
        ta_fence_after();
        if (ok) add(mine + 2u * BN);
        ta_fence_before();
    }
    __syncthreads();
    int any = 0;
    if (warp == PF_SPLITTERS + PF_DRAINERS) {
        ta_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(COLS));
    } else if (warp >= PF_SPLITTERS) {
        const int mine = quarter * 32 + lane, row = m0 + mine;
        if (row < T) {                                   // (what is computed again is stored again behind the barrier below)
            float* o = out + (size_t)row * N + n0;
            if (n0 + BN <= N && N % 4 == 0) {
#pragma unroll
                for (int j = 0; j < BN; j += 4) *reinterpret_cast<float4*>(o + j) = make_float4(sums[j], sums[j + 1], sums[j + 2], sums[j + 3]);
            } else {
#pragma unroll
                for (int j = 0; j < BN; ++j)
                    if (n0 + j < N) o[j] = sums[j];
            }
        }
        const float most_x = most[mine];
        uint32_t odd[BN / 32];
#pragma unroll
        for (int p = 0; p < BN / 32; ++p) odd[p] = 0u;
        // first all of a row's cells at once, against the largest value of any column: nearly always that is all
        float most_w = most[PF_ROWS + lane], least[4], top[4];
        if (BN > 32) most_w = pf_max_nan(most_w, most[PF_ROWS + BN - 32 + lane]);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) most_w = pf_max_nan(most_w, __shfl_xor_sync(0xffffffffu, most_w, o));
        if (n0 + BN > N) {                               // (cells of no column: some value that is in order)
#pragma unroll
            for (int j = 0; j < BN; ++j) sums[j] = n0 + j < N ? sums[j] : 1.f;
        }
#pragma unroll
        for (int j = 0; j < BN; ++j) {                   // (four chains)
            least[j % 4] = j < 4 ? fabsf(sums[j]) : fminf(least[j % 4], fabsf(sums[j]));
            top[j % 4] = j < 4 ? fabsf(sums[j]) : pf_max_nan(top[j % 4], fabsf(sums[j]));
        }
        const bool fine = (most_x < PF_LARGEST) & (most_w < PF_LARGEST) & !gave_up & (pf_max_nan(pf_max_nan(top[0], top[1]), pf_max_nan(top[2], top[3])) < INFINITY) &
                          (fminf(fminf(least[0], least[1]), fminf(least[2], least[3])) >= pf_smallest(K, most_x, most_w));
        if (!fine && row < T) {
#pragma unroll
            for (int j = 0; j < BN; ++j) {
                const float w = most[PF_ROWS + j], size = fabsf(sums[j]);
                const bool zeros = (most_x == 0.f) | (w == 0.f), whole = (size >= pf_smallest(K, most_x, w)) & (size < INFINITY);
                if (!((most_x < PF_LARGEST) & (w < PF_LARGEST) & (zeros | whole)) | (gave_up != 0)) odd[j / 32] |= 1u << (j % 32);
            }
        }
#pragma unroll
        for (int p = 0; p < BN / 32; ++p) {
            const int n = min(32, N - n0 - 32 * p);
            odd[p] = row < T && n > 0 ? odd[p] & (0xffffffffu >> (32 - n)) : 0u;
            again[mine][p] = odd[p];
            any |= odd[p] != 0u;
        }
    }
    if (!__syncthreads_or(any)) return;
    for (int r = warp; r < PF_ROWS; r += PF_THREADS / 32) {      // the cells that are computed again, a warp each
#pragma unroll 1
        for (int p = 0; p < BN / 32; ++p)
            for (uint32_t left = again[r][p]; left != 0u; left &= left - 1u) {
                const int n = n0 + 32 * p + __ffs(left) - 1;
                const float4 *xr = reinterpret_cast<const float4*>(x + (size_t)(m0 + r) * ldx), *wr = reinterpret_cast<const float4*>(W + (size_t)n * K);
                float s = 0.f;
                for (int k = lane; k < K / 4; k += 32) {
                    const float4 a = __ldg(xr + k), b = __ldg(wr + k);
                    s = fmaf(a.x, b.x, s); s = fmaf(a.y, b.y, s); s = fmaf(a.z, b.z, s); s = fmaf(a.w, b.w, s);
                }
                s = vm_warp_sum(s);
                if (lane == 0) out[(size_t)(m0 + r) * N + n] = s;
            }
    }
}

template <int BN>
int launch_products(const float* x, long long ldx, const float* W, float* out, int T, int N, int K, cudaStream_t stream) {
    const size_t smem = (size_t)PF_STAGES * 3 * (PF_ROWS + BN) * PF_K * 2;
    static VmOncePerDevice once;
    const cudaError_t e = vm_allow_smem(once, products_f32_kernel<BN>, smem);
    if (e != cudaSuccess) return (int)e;
    vm_launch_pdl(products_f32_kernel<BN>, dim3((N + BN - 1) / BN, (T + PF_ROWS - 1) / PF_ROWS), dim3(PF_THREADS), smem, stream, x, ldx, W, out, T, N, K);
    return vm_launch_status();
}

// Columns of a CTA: the fewest values split one after another on an SM, waves times rows and columns.
int choose_columns(int T, int N) {
    const int sms = vm_sm_count() > 0 ? vm_sm_count() : 1, rows = T < PF_ROWS ? T : PF_ROWS;
    long long best = 0;
    int bn = 32;
    for (int c = 32; c <= 64; c += 32) {
        const long long ctas = (long long)((T + PF_ROWS - 1) / PF_ROWS) * ((N + c - 1) / c), cost = (ctas + sms - 1) / sms * (rows + c);
        if (best == 0 || cost < best) { best = cost; bn = c; }
    }
    return bn;
}

}  // namespace

// 1 where vm_products_f32 is the faster one (see above); it takes fewer rows and cells too
VM_API int vm_products_f32_pays(int T, int N) { return T > 32 && (long long)T * N >= 350000 ? 1 : 0; }

// 1 if vm_products_f32 takes these rows (whole 16-byte pieces)
VM_API int vm_products_f32_fits(const void* x, long long ldx, const void* w, const void* out, int T, int K) {
    return T >= 1 && T <= 65535 * PF_ROWS && K > 0 && K % 4 == 0 && ldx % 4 == 0 && reinterpret_cast<uintptr_t>(x) % 16 == 0 &&
                   reinterpret_cast<uintptr_t>(w) % 16 == 0 && reinterpret_cast<uintptr_t>(out) % 16 == 0
               ? 1
               : 0;
}

// x float32 [T, K] with rows ldx apart, w float32 [N, K], out float32 [T, N]
VM_API int vm_products_f32(const float* x, long long ldx, const float* w, float* out, int T, int N, int K, cudaStream_t stream) {
    if (T <= 0 || N <= 0) return 0;
    if (!vm_products_f32_fits(x, ldx, w, out, T, K)) return VM_ERR_UNSUPPORTED;
    switch (choose_columns(T, N)) {
        case 32: return launch_products<32>(x, ldx, w, out, T, N, K, stream);
        default: return launch_products<64>(x, ldx, w, out, T, N, K, stream);
    }
}
