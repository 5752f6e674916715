// Decode attention in bfloat16 with every option of attention_biased.cu (bias by bucketed distance, slopes, sink, window, kept first
// tokens, chunked mask, values inside the key rows): each sequence brings ONE new token, and its query heads read the cache.
//
// What bounds it is latency: a few hundred keys of a few sequences are a microsecond of memory traffic.  A CTA with a warp's lanes as keys
// read every key row once per query head, and summed the values of 32 keys one after another (8 sequences, 16 heads on 4 kv heads, 700
// cached tokens: 21 us; two of 32 heads over one latent of 160 values, 2,000 cached tokens: 78 us).  Here the query heads of a kv
// head are the rows of an mma.sync tile (up to 16), a warp takes 32 keys at a time, and all of a warp's loads go straight from global memory
// into the registers the tensor cores read: 16 bytes each, all in flight together, no staging and no barrier before the sums meet.
//   * Q K^T: the contraction may run in any order, so lane (g, t) takes 8 neighbouring values of key g's row (and of query g's) as the
//     operands of two products, instead of the 2 + 2 that the instruction's own order would give it.
//   * P V: lane (g, t) takes 8 neighbouring columns of four value rows and pairs them up byte by byte; column j of its eight is the
//     n = g of product j, so the sums come out in an order that the last step undoes.
// The probabilities stay 32 bits wide: each is the exact sum of three bfloat16 parts, and the three products go into the same float32
// sum.  (An infinite value meets the first part alone: 0 times it would not be a number.)
//
// The keys of a (sequence, kv head) go to the warps of `splits` CTAs in turn, 32 at a time from absolute multiples of 32.  A CTA's warps
// meet in shared memory, the CTAs (a thread-block cluster) in each other's: every CTA finishes its share of the outputs, one hardware
// barrier, no scratch in global memory and no counters.  How many CTAs share a sequence follows from the step's shape (sequences, heads, table
// width), and with it the order of a token's sums: its last bits are not the same in every batch.  Measured in a step: 6.7 us and
// 10.0 us for the two shapes above.
#include <algorithm>

#include "mma.cuh"

namespace {

constexpr int WARPS = 8;
constexpr int ROWS = 16;                 // query heads of a CTA
constexpr int KEYS = 32;                 // keys of a warp's turn
constexpr int MAX_SPLITS = 8;            // CTAs of a portable cluster

__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
// one float into the shared memory of the cluster's CTA `rank`, at the place that `local` has in this CTA's own
__device__ __forceinline__ void store_to(int rank, float* local, float v) {
    unsigned at;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"((unsigned)__cvta_generic_to_shared(local)), "r"(rank));
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(at), "f"(v) : "memory");
}

// a bias, slope or sink in the softmax's base-2 units; a finite one stays finite (the lowest float, as masks use it, times log2(e) is not, and a row whose
// keys all carry it would have no largest score)
__device__ __forceinline__ float base2(float v) {
    const float y = v * 1.4426950408889634f;
    return isinf(y) && !isinf(v) ? copysignf(3.402823466e38f, v) : y;
}

// two bfloat16 with every infinity and NaN replaced by zero
__device__ __forceinline__ unsigned finite_only(unsigned v) {
    const unsigned bad = __vcmpeq2(v & 0x7f807f80u, 0x7f807f80u);
    return v & ~bad;
}

// p = hi + mid + lo exactly, each part a bfloat16 (round to nearest leaves a rest of at most 16, then 8 bits)
__device__ __forceinline__ void three_parts(float p0, float p1, unsigned& hi, unsigned& mid, unsigned& lo) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(p0, p1);
    const float2 hf = __bfloat1622float2(h);
    const float r0 = p0 - hf.x, r1 = p1 - hf.y;
    const __nv_bfloat162 m = __floats2bfloat162_rn(r0, r1);
    const float2 mf = __bfloat1622float2(m);
    hi = *reinterpret_cast<const unsigned*>(&h);
    mid = *reinterpret_cast<const unsigned*>(&m);
    lo = vm_pack_bf16(r0 - mf.x, r1 - mf.y);
}

template <int DV> constexpr int row_floats() { return DV + 8; }      // a result row: DV sums, maximum, denominator; 8 banks from row to row

template <int DK, int DV>
__global__ void __launch_bounds__(WARPS * 32, 1)
attn_decode_tile_kernel(const __nv_bfloat16* __restrict__ q, int q_row_stride, const __nv_bfloat16* __restrict__ kpages,
                        const __nv_bfloat16* __restrict__ vpages, const int* __restrict__ block_table, int max_blocks,
                        const int* __restrict__ positions, const float* __restrict__ rel, const int* __restrict__ bucket_of, int far,
                        __nv_bfloat16* __restrict__ out, int H, int Hkv, float scale_log2, int window, int keep_first, int chunk, int n_pages,
                        const float* __restrict__ sink, const float* __restrict__ slopes, int v_stride, int* __restrict__ err) {
    constexpr int RF = row_floats<DV>(), KB = DK / 32, VH = DV / 64;
    extern __shared__ __align__(16) float part[];          // [WARPS][ROWS][RF]; with splits also [splits][share of the outputs]
    __shared__ float fac[WARPS][ROWS], row_top[MAX_SPLITS][ROWS], row_sum[MAX_SPLITS][ROWS];
    const int split = blockIdx.x, splits = gridDim.x, b = blockIdx.z;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t4 = lane & 3;
    const int G = H / Hkv, per_kv = (G + ROWS - 1) / ROWS;
    const int hk = blockIdx.y / per_kv, first = (blockIdx.y - hk * per_kv) * ROWS;
    const int h0 = hk * G + first, ng = min(ROWS, G - first);
    vm_pdl_launch_dependents();
    if (splits > 1) cluster_arrive();                      // every CTA has started before anyone writes into it
    vm_pdl_wait();
    const int pos = positions[b];
    const int lo = vm_first_seen(pos, window, chunk);
    const int kept = min(keep_first, lo);
    const int first_chunk = lo / KEYS, kept_chunks = min((kept + KEYS - 1) / KEYS, first_chunk);
    const int n_chunks = kept_chunks + pos / KEYS - first_chunk + 1;
    const int* table = block_table + (size_t)b * max_blocks;
    auto base_of = [&](int c) { return (c < kept_chunks ? c : first_chunk + (c - kept_chunks)) * KEYS; };
    auto page_of = [&](int base) { const int blk = base / VM_PAGE_TOKENS; return blk < max_blocks ? table[blk] : -1; };
    int c = split * WARPS + warp;
    int page = c < n_chunks ? page_of(base_of(c)) : -1;

    // the queries: row g and row g + 8 of the tile, 8 neighbouring values a lane
    uint4 qa[KB], qb[KB];
    {
        const __nv_bfloat16* row = q + (size_t)b * q_row_stride + (size_t)h0 * DK + t4 * 8;
#pragma unroll
        for (int kb = 0; kb < KB; ++kb) {
            qa[kb] = g < ng ? *reinterpret_cast<const uint4*>(row + (size_t)g * DK + kb * 32) : make_uint4(0u, 0u, 0u, 0u);
            qb[kb] = g + 8 < ng ? *reinterpret_cast<const uint4*>(row + (size_t)(g + 8) * DK + kb * 32) : make_uint4(0u, 0u, 0u, 0u);
        }
    }
    const float slope_a = slopes && g < ng ? base2(slopes[h0 + g]) : 0.f, slope_b = slopes && g + 8 < ng ? base2(slopes[h0 + g + 8]) : 0.f;
    float m_a = -INFINITY, m_b = -INFINITY, l_a = 0.f, l_b = 0.f;
    float o[VH * 8][4];
#pragma unroll
    for (int i = 0; i < VH * 8; ++i) o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.f;

    for (; c < n_chunks; c += splits * WARPS) {
        const int base = base_of(c);
        if (page < 0 || page >= n_pages) {                 // a page the step needs is not there: report, skip
            if (lane == 0 && err) atomicExch(err, VM_ERRWORD_CACHE_READ);
            page = c + splits * WARPS < n_chunks ? page_of(base_of(c + splits * WARPS)) : -1;
            continue;
        }
        const size_t tok0 = ((size_t)page * Hkv + hk) * VM_PAGE_TOKENS + (base % VM_PAGE_TOKENS);
        auto sees = [&](int key) { return key <= pos && (key >= lo || key < kept); };
        // ---- every load of the turn; keys that are not seen (their rows may hold anything) read as zeros
        uint4 kf[4][KB];
#pragma unroll
        for (int nb = 0; nb < 4; ++nb) {
            const int key = nb * 8 + g;
            const bool ok = sees(base + key);
            const __nv_bfloat16* row = kpages + (tok0 + key) * DK + t4 * 8;
#pragma unroll
            for (int kb = 0; kb < KB; ++kb) kf[nb][kb] = ok ? *reinterpret_cast<const uint4*>(row + kb * 32) : make_uint4(0u, 0u, 0u, 0u);
        }
        uint4 vf[2][4][VH];
        auto load_values = [&]() {
#pragma unroll
            for (int ks = 0; ks < 2; ++ks)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int key = ks * 16 + 2 * t4 + (e & 1) + 8 * (e >> 1);
                    const bool ok = sees(base + key);
                    const __nv_bfloat16* row = vpages + (tok0 + key) * v_stride + g * 8;
#pragma unroll
                    for (int vh = 0; vh < VH; ++vh) vf[ks][e][vh] = ok ? *reinterpret_cast<const uint4*>(row + vh * 64) : make_uint4(0u, 0u, 0u, 0u);
                }
        };
        if (DK + DV <= 192) load_values();                 // (with wider rows the registers hold keys first and values then)
        float bias[4][4];
        if (rel) {
#pragma unroll
            for (int nb = 0; nb < 4; ++nb)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int away = pos - (base + nb * 8 + 2 * t4 + e);
                    const float* row = rel + (size_t)bucket_of[min(max(away, 0), far)] * H + h0;
                    bias[nb][e] = g < ng ? base2(row[g]) : 0.f;
                    bias[nb][2 + e] = g + 8 < ng ? base2(row[g + 8]) : 0.f;
                }
        }
        page = c + splits * WARPS < n_chunks ? page_of(base_of(c + splits * WARPS)) : -1;
        // ---- scores
        float s[4][4];
#pragma unroll
        for (int nb = 0; nb < 4; ++nb) {
            s[nb][0] = s[nb][1] = s[nb][2] = s[nb][3] = 0.f;
#pragma unroll
            for (int kb = 0; kb < KB; ++kb) {
                vm_mma_bf16_16816(s[nb], qa[kb].x, qb[kb].x, qa[kb].y, qb[kb].y, kf[nb][kb].x, kf[nb][kb].y);
                vm_mma_bf16_16816(s[nb], qa[kb].z, qb[kb].z, qa[kb].w, qb[kb].w, kf[nb][kb].z, kf[nb][kb].w);
            }
        }
        if (DK + DV > 192) load_values();
        float mx_a = -INFINITY, mx_b = -INFINITY;
#pragma unroll
        for (int nb = 0; nb < 4; ++nb)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int key = base + nb * 8 + 2 * t4 + e;
                const float away = (float)(pos - key);
                const float ba = fmaf(-slope_a, away, rel ? bias[nb][e] : 0.f), bb = fmaf(-slope_b, away, rel ? bias[nb][2 + e] : 0.f);
                const bool ok = sees(key);
                s[nb][e] = ok ? fmaf(s[nb][e], scale_log2, ba) : -INFINITY;
                s[nb][2 + e] = ok ? fmaf(s[nb][2 + e], scale_log2, bb) : -INFINITY;
                mx_a = fmaxf(mx_a, s[nb][e]);
                mx_b = fmaxf(mx_b, s[nb][2 + e]);
            }
        mx_a = fmaxf(mx_a, __shfl_xor_sync(0xffffffffu, mx_a, 1)); mx_a = fmaxf(mx_a, __shfl_xor_sync(0xffffffffu, mx_a, 2));
        mx_b = fmaxf(mx_b, __shfl_xor_sync(0xffffffffu, mx_b, 1)); mx_b = fmaxf(mx_b, __shfl_xor_sync(0xffffffffu, mx_b, 2));
        const float top_a = fmaxf(m_a, mx_a), top_b = fmaxf(m_b, mx_b);
        const float use_a = top_a == -INFINITY ? 0.f : top_a, use_b = top_b == -INFINITY ? 0.f : top_b;
        const float al_a = exp2f(m_a - use_a), al_b = exp2f(m_b - use_b);
        m_a = top_a; m_b = top_b;
        l_a *= al_a; l_b *= al_b;
#pragma unroll
        for (int i = 0; i < VH * 8; ++i) { o[i][0] *= al_a; o[i][1] *= al_a; o[i][2] *= al_b; o[i][3] *= al_b; }
        // ---- P V, 16 keys at a time: rows of P in three exact parts, values paired up
#pragma unroll
        for (int ks = 0; ks < 2; ++ks) {
            unsigned ph[4], pm[4], pl[4];
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                float* x = s[2 * ks + half];
                const float p0 = exp2f(x[0] - use_a), p1 = exp2f(x[1] - use_a), p2 = exp2f(x[2] - use_b), p3 = exp2f(x[3] - use_b);
                l_a += p0 + p1; l_b += p2 + p3;
                three_parts(p0, p1, ph[2 * half], pm[2 * half], pl[2 * half]);
                three_parts(p2, p3, ph[2 * half + 1], pm[2 * half + 1], pl[2 * half + 1]);
            }
#pragma unroll
            for (int vh = 0; vh < VH; ++vh) {
                const unsigned* v0 = reinterpret_cast<const unsigned*>(&vf[ks][0][vh]);
                const unsigned* v1 = reinterpret_cast<const unsigned*>(&vf[ks][1][vh]);
                const unsigned* v2 = reinterpret_cast<const unsigned*>(&vf[ks][2][vh]);
                const unsigned* v3 = reinterpret_cast<const unsigned*>(&vf[ks][3][vh]);
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const unsigned pick = (j & 1) ? 0x7632u : 0x5410u;
                    const unsigned b0 = __byte_perm(v0[j / 2], v1[j / 2], pick), b1 = __byte_perm(v2[j / 2], v3[j / 2], pick);
                    const unsigned f0 = finite_only(b0), f1 = finite_only(b1);
                    float* acc = o[vh * 8 + j];
                    vm_mma_bf16_16816(acc, pl[0], pl[1], pl[2], pl[3], f0, f1);
                    vm_mma_bf16_16816(acc, pm[0], pm[1], pm[2], pm[3], f0, f1);
                    vm_mma_bf16_16816(acc, ph[0], ph[1], ph[2], ph[3], b0, b1);
                }
            }
        }
    }
    // ---- this warp's rows
    l_a += __shfl_xor_sync(0xffffffffu, l_a, 1); l_a += __shfl_xor_sync(0xffffffffu, l_a, 2);
    l_b += __shfl_xor_sync(0xffffffffu, l_b, 1); l_b += __shfl_xor_sync(0xffffffffu, l_b, 2);
    {
        float* ra = part + (size_t)(warp * ROWS + g) * RF;
        float* rb = ra + 8 * RF;
        if (g < ng) {
#pragma unroll
            for (int i = 0; i < VH * 8; ++i) *reinterpret_cast<float2*>(ra + i * 8 + 2 * t4) = make_float2(o[i][0], o[i][1]);
            if (t4 == 0) { ra[DV] = m_a; ra[DV + 1] = l_a; }
        }
        if (g + 8 < ng) {
#pragma unroll
            for (int i = 0; i < VH * 8; ++i) *reinterpret_cast<float2*>(rb + i * 8 + 2 * t4) = make_float2(o[i][2], o[i][3]);
            if (t4 == 0) { rb[DV] = m_b; rb[DV + 1] = l_b; }
        }
    }
    __syncthreads();
    if (splits > 1) cluster_wait();
    // the warps' factors; the CTA's maximum and denominator of every row, for every CTA of the cluster
    if (threadIdx.x < WARPS * ROWS) {
        const int w = threadIdx.x / ROWS, r = threadIdx.x % ROWS;
        if (r < ng) {
            float m[WARPS], M = -INFINITY;
#pragma unroll
            for (int i = 0; i < WARPS; ++i) { m[i] = part[(size_t)(i * ROWS + r) * RF + DV]; M = fmaxf(M, m[i]); }
            const float use = M == -INFINITY ? 0.f : M;    // (a warp without keys: factor 0)
            fac[w][r] = exp2f(part[(size_t)(w * ROWS + r) * RF + DV] - use);
            if (w == 0) {
                float L = 0.f;
#pragma unroll
                for (int i = 0; i < WARPS; ++i) L = fmaf(part[(size_t)(i * ROWS + r) * RF + DV + 1], exp2f(m[i] - use), L);
                if (splits == 1) { row_top[0][r] = M; row_sum[0][r] = L; }
                else for (int to = 0; to < splits; ++to) { store_to(to, &row_top[split][r], M); store_to(to, &row_sum[split][r], L); }
            }
        }
    }
    __syncthreads();
    // output i of the CTA's heads (row i / DV, column d = i % DV, which lies at: 64-column half, then d % 8, then (d / 8) % 8) over its warps
    auto sum = [&](int i) {
        const int r = i / DV, d = i % DV;
        const float* col = part + (size_t)r * RF + (d & ~63) + (d & 7) * 8 + ((d >> 3) & 7);
        float acc = 0.f;
#pragma unroll
        for (int w = 0; w < WARPS; ++w) acc = fmaf(col[(size_t)w * ROWS * RF], fac[w][r], acc);
        return acc;
    };
    const int total = ng * DV, share = (total + splits - 1) / splits;
    float* got = part + WARPS * ROWS * RF;                 // [splits][share]
    if (splits > 1) {
        for (int i = threadIdx.x; i < total; i += WARPS * 32) {
            const int owner = i / share;
            store_to(owner, got + split * share + (i - owner * share), sum(i));
        }
        cluster_arrive();
        cluster_wait();
    }
    for (int i = split * share + threadIdx.x; i < min(total, (split + 1) * share); i += WARPS * 32) {
        const int r = i / DV, d = i % DV;
        float M = row_top[0][r], L = row_sum[0][r], acc = 0.f;
        if (splits == 1) {
            acc = sum(i);
        } else {
            for (int c2 = 1; c2 < splits; ++c2) M = fmaxf(M, row_top[c2][r]);
            const float use = M == -INFINITY ? 0.f : M;
            L = 0.f;
            for (int c2 = 0; c2 < splits; ++c2) {
                const float f = exp2f(row_top[c2][r] - use);
                acc = fmaf(got[c2 * share + i - split * share], f, acc);
                L = fmaf(row_sum[c2][r], f, L);
            }
        }
        float keep = 1.f;
        if (sink) {                                        // exp(sink): one more term of the denominator, without a value
            const float sk = base2(sink[h0 + r]), top = fmaxf(M, sk);
            keep = exp2f(M - top);
            L = L * keep + exp2f(sk - top);
        }
        out[((size_t)b * H + h0 + r) * DV + d] = __float2bfloat16_rn(acc * (keep / L));
    }
}

template <int DK, int DV>
int launch_tile(const void* q, int q_row_stride, const void* kpages, const void* vpages, const int* block_table, int max_blocks, const int* positions,
                const float* rel, const int* bucket_of, int far, const float* sink, const float* slopes, int v_stride, void* out, int B, int H, int Hkv,
                float scale, int window, int keep_first, int chunk, int n_pages, int* err, cudaStream_t stream) {
    const int G = H / Hkv, groups = Hkv * ((G + ROWS - 1) / ROWS);
    // CTAs of a (sequence, head group): enough for one turn of every warp (measured: a second turn costs 1.7 us with keys of 64 and 4 us with keys of
    // 128 and more, a cluster of two or four instead of one CTA 2 us), as far as the GPU has SMs for them all; clusters of eight only for at most
    // 64 CTAs (a cluster lies inside a GPC: sixteen of them are not resident at once, and 128 CTAs took 11.4 us where clusters of four take 8.4).  From
    // the step's shape alone (the block table's width, the masks), so that a recorded launch stays valid as sequences grow
    long long keys = (long long)max_blocks * VM_PAGE_TOKENS;
    if (window > 0) keys = std::min<long long>(keys, window + (long long)keep_first + 2 * KEYS);
    if (chunk > 0) keys = std::min<long long>(keys, chunk + (long long)keep_first + 2 * KEYS);
    const long long tiles = (long long)B * groups;
    int splits = 1;
    while (splits < MAX_SPLITS && 2 * splits * tiles <= (splits == 4 ? 64 : vm_sm_count()) && (long long)splits * WARPS * KEYS < keys) splits *= 2;
    const size_t smem = ((size_t)WARPS * ROWS * row_floats<DV>() + (splits > 1 ? ROWS * DV + splits : 0)) * sizeof(float);
    static VmOncePerDevice once;
    const cudaError_t allowed = vm_allow_smem(once, attn_decode_tile_kernel<DK, DV>, (WARPS * ROWS * row_floats<DV>() + ROWS * DV + MAX_SPLITS) * sizeof(float));
    if (allowed != cudaSuccess) return (int)allowed;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(splits, groups, B);
    cfg.blockDim = dim3(WARPS * 32);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = splits; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = vm_pdl_enabled ? 2 : 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, attn_decode_tile_kernel<DK, DV>, (const __nv_bfloat16*)q, q_row_stride, (const __nv_bfloat16*)kpages,
                                             (const __nv_bfloat16*)vpages, block_table, max_blocks, positions, rel, bucket_of, far, (__nv_bfloat16*)out, H, Hkv,
                                             scale * 1.4426950408889634f, window, keep_first, chunk, n_pages, sink, slopes, v_stride, err);
    const int status = vm_launch_status();
    return status ? status : (int)e;
}

bool aligned16(const void* p) { return reinterpret_cast<uintptr_t>(p) % 16 == 0; }

}  // namespace

// 1 if vm_attention_decode_tile takes these sizes and rows: the instantiated head sizes, 16-byte rows
VM_API int vm_attention_decode_tile_fits(const void* q, int q_row_stride, const void* kpages, const void* vpages, int B, int H, int Hkv, int Dk, int Dv,
                                         int v_stride) {
    const bool sizes = (Dv == 64 && (Dk == 64 || Dk == 96 || Dk == 128)) || (Dv == 128 && (Dk == 64 || Dk == 96 || Dk == 128 || Dk == 160 || Dk == 192));
    return sizes && H > 0 && Hkv > 0 && H % Hkv == 0 && q_row_stride % 8 == 0 && v_stride % 8 == 0 && v_stride >= Dv && aligned16(q) && aligned16(kpages) &&
                   aligned16(vpages) && B <= 65535 && (long long)Hkv * ((H / Hkv + ROWS - 1) / ROWS) <= 65535
               ? 1
               : 0;
}

// one new token per sequence (token s belongs to sequence s); arguments as vm_attention_sink_decode_bf16, v_stride given
VM_API int vm_attention_decode_tile(const void* q, int q_row_stride, const void* kpages, const void* vpages, const int* block_table, int max_blocks,
                                    const int* positions, const float* rel, const int* bucket_of, int far, const float* sink, const float* slopes,
                                    int v_stride, void* out, int B, int H, int Hkv, int Dk, int Dv, float scale, int window, int keep_first, int chunk,
                                    int n_pages, int* err, cudaStream_t stream) {
    if (B <= 0) return 0;
    if (!vm_attention_decode_tile_fits(q, q_row_stride, kpages, vpages, B, H, Hkv, Dk, Dv, v_stride)) return VM_ERR_UNSUPPORTED;
#define VM_TILE(K, V)                                                                                                                            \
    if (Dk == K && Dv == V)                                                                                                                      \
        return launch_tile<K, V>(q, q_row_stride, kpages, vpages, block_table, max_blocks, positions, rel, bucket_of, far, sink, slopes, v_stride, out, B, \
                                 H, Hkv, scale, window, keep_first, chunk, n_pages, err, stream);
    VM_TILE(64, 64) VM_TILE(96, 64) VM_TILE(128, 64)
    VM_TILE(64, 128) VM_TILE(96, 128) VM_TILE(128, 128) VM_TILE(160, 128) VM_TILE(192, 128)
#undef VM_TILE
    return VM_ERR_UNSUPPORTED;
}
