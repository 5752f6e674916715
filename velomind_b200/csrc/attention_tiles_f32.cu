// Attention over the paged cache in float32 for prompts: the arithmetic of attention_rows.cu, bit for bit, with neighbouring tokens of a head in one CTA that
// walk the keys together.  Options as there: a bias by bucketed distance, slopes, a sink, a window with kept first tokens, a chunked mask, values inside the
// key rows.
//
// In attention_rows.cu a CTA owns up to eight query rows and its eight warps share the keys, which is right for a few rows: a prompt's CTAs find work for two or
// three of the warps (a prompt of 190 tokens has six chunks of 32 keys at its end and one at its start), every one of them fetches its chunk for eight rows
// alone, and what bounds them is the chain of a warp that has nothing beside it.  Here a CTA of four warps owns 4 R tokens of a head; a warp has R of them as
// rows, one key per lane, and all four use a chunk that was fetched once, while the next one is on its way (asynchronous copies, two buffers).
//
// Measured, 9 heads of 64, that kernel / this one: four prompts of 33 to 190 tokens 57.9 / 24.7 us, one of 446 74 / 48, of 2,048 779 / 472, sixteen of 16 14.2 / 6.0;
// 16 heads, four of 33 to 190 74 / 33.6.  Small steps stay with that kernel (one of 64 tokens 5.7 / 8.6), and new tokens behind a long prefix, whose keys its warps
// share (40 tokens behind 1,000 27 / 79).
//
// The sums keep their order: chunk c belongs to class c mod 8, a class has a maximum, a denominator and sums of its own (in shared memory between its chunks),
// and the classes meet in their order at the end, as the eight warps of the other kernel do.
#include "mma.cuh"

namespace {

constexpr int TF_WARPS = 4, TF_KEYS = 32, TF_CLASSES = 8;

__host__ __device__ constexpr int tf_pitch(int Dk) { return Dk + (Dk % 8 == 0 ? 4 : 8); }      // floats of a key row: an odd number of 16-byte units
__host__ __device__ constexpr int tf_classes(int max_blocks) { return 2 * max_blocks < TF_CLASSES ? 2 * max_blocks : TF_CLASSES; }      // (that the table has chunks for)
__host__ __device__ constexpr size_t tf_bytes(int R, int Dk, int Dv, int classes) {
    return sizeof(float) * ((size_t)2 * TF_KEYS * (tf_pitch(Dk) + Dv) + (size_t)TF_WARPS * R * (Dk + TF_KEYS) + (size_t)classes * TF_WARPS * R * (Dv + 2));
}
constexpr size_t TF_MOST_BYTES = 200 * 1024;

// R: rows of a warp; VP: pairs of value columns per lane, 2 lane + 64 i and the next
template <int R, int VP>
__global__ void __launch_bounds__(TF_WARPS * 32)
attn_tiles_f32_kernel(const float* __restrict__ q, int q_row_stride, const float* __restrict__ kpages, const float* __restrict__ vpages,
                      const int* __restrict__ block_table, int max_blocks, const int* __restrict__ positions, const int* __restrict__ seq_of_token,
                      const float* __restrict__ rel, const int* __restrict__ bucket_of, int far, float* __restrict__ out, int n_tokens, int H, int Hkv, int Dk,
                      int Dv, float scale, int window, int keep_first, int chunk, int n_pages, const float* __restrict__ sink,
                      const float* __restrict__ slopes, int v_stride, int* __restrict__ err) {
    constexpr int TILE = TF_WARPS * R;
    extern __shared__ __align__(16) float sm[];
    const int KP = tf_pitch(Dk), SP = Dv + 2;
    float* sk = sm;                                        // [2][32][KP]
    float* sv = sk + 2 * TF_KEYS * KP;                     // [2][32][Dv]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    float* sq = sv + 2 * TF_KEYS * Dv + warp * R * Dk;     // [R][Dk] the warp's scaled queries
    float* sp = sv + 2 * TF_KEYS * Dv + TF_WARPS * R * Dk + warp * R * TF_KEYS;             // [R][32] its probabilities
    float* state = sv + 2 * TF_KEYS * Dv + TF_WARPS * R * (Dk + TF_KEYS) + (size_t)warp * tf_classes(max_blocks) * R * SP;      // [classes][R][sums, maximum, denominator]
    const int h = blockIdx.y, hk = h / (H / Hkv);
    const int t0 = ((int)gridDim.x - 1 - (int)blockIdx.x) * TILE, n_here = min(TILE, n_tokens - t0);      // (the longest rows first)
    const int my_seq = lane < n_here ? seq_of_token[t0 + lane] : -1, my_pos = lane < n_here ? positions[t0 + lane] : -1;
    const int my_lo = vm_first_seen(my_pos, window, chunk);
    // the 16-byte units of a chunk that this thread copies: its first, and how far apart they are, in rows and units
    const int ku = Dk / 4, vu = Dv / 4;
    const int k_row = threadIdx.x / ku, k_col = threadIdx.x % ku, k_rows = TF_WARPS * 32 / ku, k_cols = TF_WARPS * 32 % ku;
    const int v_row = threadIdx.x / vu, v_col = threadIdx.x % vu, v_rows = TF_WARPS * 32 / vu, v_cols = TF_WARPS * 32 % vu;

    for (int i = lane; i < R * Dk; i += 32) {
        const int r = i / Dk, d = i - r * Dk, t = warp * R + r;
        sq[i] = t < n_here ? q[(size_t)(t0 + t) * q_row_stride + (size_t)h * Dk + d] * scale : 0.f;
    }
    for (int start = 0; start < n_here;) {
        // the neighbouring tokens of one sequence (a tile may cross into the next one: another turn)
        const int seq = __shfl_sync(0xffffffffu, my_seq, start);
        const unsigned others = __ballot_sync(0xffffffffu, lane > start && (lane >= n_here || my_seq != seq));
        const int end = others ? __ffs(others) - 1 : n_here;
        const bool in = lane >= start && lane < end;
        const int lowest = __reduce_min_sync(0xffffffffu, in ? my_lo : 0x7fffffff), highest = __reduce_max_sync(0xffffffffu, in ? my_pos : -1);
        const int kept_most = __reduce_max_sync(0xffffffffu, in ? min(keep_first, my_lo) : 0);
        const int warp_highest = __reduce_max_sync(0xffffffffu, in && lane / R == warp ? my_pos : -1);
        int pos[R], lo[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int t = warp * R + r;
            pos[r] = __shfl_sync(0xffffffffu, my_pos, t); lo[r] = __shfl_sync(0xffffffffu, my_lo, t);
            if (t < start || t >= end) { pos[r] = -1; lo[r] = 0x7fffffff; }      // a row that is not there sees nothing
        }
        auto next_chunk = [&](int c) { return c * 32 >= kept_most && c < lowest / 32 ? lowest / 32 : c; };      // not between the kept tokens and the window
        auto page_of = [&](int c) {
            const int blk = c * 32 / VM_PAGE_TOKENS;
            return c * 32 <= highest && blk < max_blocks ? block_table[(size_t)seq * max_blocks + blk] : -1;
        };
        auto fetch = [&](int c, int page, int buf) {       // a chunk's keys and values into a buffer
            if (c * 32 <= highest && page >= 0 && page < n_pages) {
                const size_t tok0 = ((size_t)page * Hkv + hk) * VM_PAGE_TOKENS + (c * 32 % VM_PAGE_TOKENS);
                const int rows = min(TF_KEYS, highest - c * 32 + 1);
                float* dk = sk + buf * TF_KEYS * KP;
                float* dv = sv + buf * TF_KEYS * Dv;
                for (int row = k_row, col = k_col; row < rows;) {
                    vm_cp_async16(dk + row * KP + 4 * col, kpages + (tok0 + row) * Dk + 4 * col);
                    row += k_rows; col += k_cols;
                    if (col >= ku) { col -= ku; ++row; }
                }
                for (int row = v_row, col = v_col; row < rows;) {
                    vm_cp_async16(dv + row * Dv + 4 * col, vpages + (tok0 + row) * v_stride + 4 * col);
                    row += v_rows; col += v_cols;
                    if (col >= vu) { col -= vu; ++row; }
                }
            }
            vm_cp_async_commit();
        };
        int c = next_chunk(0), page = page_of(c), buf = 0;
        fetch(c, page, 0);
        int c_next = next_chunk(c + 1), page_next = page_of(c_next);
        unsigned visited = 0;                              // classes with a state
        for (; c * 32 <= highest; c = c_next, page = page_next, c_next = next_chunk(c + 1), page_next = page_of(c_next), buf ^= 1) {
            fetch(c_next, page_next, buf ^ 1);
            asm volatile("cp.async.wait_group 1;\n" ::);
            __syncthreads();                               // the chunk is there for all
            const int base = c * 32;
            if (page < 0 || page >= n_pages) {             // a page the step needs is not there: report, skip
                if (threadIdx.x == 0 && err) atomicExch(err, VM_ERRWORD_CACHE_READ);
            } else if (base <= warp_highest) {
                const int j = base + lane, cls = c % TF_CLASSES;
                const float* krow = sk + buf * TF_KEYS * KP + lane * KP;
                const float* vals = sv + buf * TF_KEYS * Dv + 2 * lane;
                float* mine = state + (size_t)cls * R * SP;
                float s[R];
#pragma unroll
                for (int r = 0; r < R; ++r) s[r] = 0.f;
#pragma unroll 4
                for (int d = 0; d < Dk; d += 4) {
                    const float4 k4 = *reinterpret_cast<const float4*>(krow + d);
#pragma unroll
                    for (int r = 0; r < R; ++r) {
                        const float4 q4 = *reinterpret_cast<const float4*>(sq + r * Dk + d);
                        s[r] = fmaf(q4.x, k4.x, s[r]); s[r] = fmaf(q4.y, k4.y, s[r]);
                        s[r] = fmaf(q4.z, k4.z, s[r]); s[r] = fmaf(q4.w, k4.w, s[r]);
                    }
                }
                // the class's state (all rows' chains side by side: nothing here waits for another row)
                float acc[R][VP][2], m[R], l[R];
                const bool again = visited >> cls & 1u;
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    m[r] = again ? mine[r * SP + Dv] : -INFINITY;
                    l[r] = again ? mine[r * SP + Dv + 1] : 0.f;
#pragma unroll
                    for (int i = 0; i < VP; ++i) {
                        const float2 a = again && 2 * lane + 64 * i < Dv ? *reinterpret_cast<const float2*>(mine + r * SP + 2 * lane + 64 * i) : make_float2(0.f, 0.f);
                        acc[r][i][0] = a.x; acc[r][i][1] = a.y;
                    }
                }
                unsigned seen[R];                          // which of the chunk's keys each row sees
                bool all_seen = true;
                float top[R], p[R], alpha[R];
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    const bool valid = j <= pos[r] && (j >= lo[r] || j < min(keep_first, lo[r]));
                    seen[r] = __ballot_sync(0xffffffffu, valid);
                    all_seen = all_seen && (pos[r] < 0 || seen[r] == 0xffffffffu);
                    if (rel && valid) s[r] += rel[(size_t)bucket_of[min(pos[r] - j, far)] * H + h];
                    if (slopes && valid) s[r] = fmaf(-slopes[h], (float)(pos[r] - j), s[r]);
                    if (!valid) s[r] = -INFINITY;
                    top[r] = s[r];
                }
#pragma unroll
                for (int o = 16; o > 0; o >>= 1)
#pragma unroll
                    for (int r = 0; r < R; ++r) top[r] = fmaxf(top[r], __shfl_xor_sync(0xffffffffu, top[r], o));
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    top[r] = fmaxf(m[r], top[r]);
                    const float use = top[r] == -INFINITY ? 0.f : top[r];      // nothing seen so far: no factor changes anything
                    p[r] = seen[r] >> lane & 1u ? expf(s[r] - use) : 0.f;
                    alpha[r] = expf(m[r] - use);
                    sp[r * TF_KEYS + lane] = p[r];
#pragma unroll
                    for (int i = 0; i < VP; ++i) { acc[r][i][0] *= alpha[r]; acc[r][i][1] *= alpha[r]; }
                }
#pragma unroll
                for (int o = 16; o > 0; o >>= 1)
#pragma unroll
                    for (int r = 0; r < R; ++r) p[r] += __shfl_xor_sync(0xffffffffu, p[r], o);
                __syncwarp();                              // (every lane has read the state, the probabilities are written)
                if (lane == 0)
#pragma unroll
                    for (int r = 0; r < R; ++r) { mine[r * SP + Dv] = top[r]; mine[r * SP + Dv + 1] = fmaf(l[r], alpha[r], p[r]); }
                const int last = min(TF_KEYS - 1, warp_highest - base);
                // values of 32 keys; at the edge of a mask a row takes the ones it sees and no others (they may hold anything, infinities too)
                if (all_seen) {
#pragma unroll 2
                    for (int jj = 0; jj < TF_KEYS; jj += 4) {
                        float2 v[4][VP];
#pragma unroll
                        for (int e = 0; e < 4; ++e)
#pragma unroll
                            for (int i = 0; i < VP; ++i) v[e][i] = 2 * lane + 64 * i < Dv ? *reinterpret_cast<const float2*>(vals + (jj + e) * Dv + 64 * i) : make_float2(0.f, 0.f);
#pragma unroll
                        for (int r = 0; r < R; ++r) {
                            const float4 p4 = *reinterpret_cast<const float4*>(sp + r * TF_KEYS + jj);
                            const float pe[4] = {p4.x, p4.y, p4.z, p4.w};
#pragma unroll
                            for (int e = 0; e < 4; ++e)
#pragma unroll
                                for (int i = 0; i < VP; ++i) {
                                    acc[r][i][0] = fmaf(pe[e], v[e][i].x, acc[r][i][0]);
                                    acc[r][i][1] = fmaf(pe[e], v[e][i].y, acc[r][i][1]);
                                }
                        }
                    }
                } else {
#pragma unroll 1
                    for (int jj = 0; jj <= last; jj += 4) {
                        float2 v[4][VP];
#pragma unroll
                        for (int e = 0; e < 4; ++e)
#pragma unroll
                            for (int i = 0; i < VP; ++i) v[e][i] = 2 * lane + 64 * i < Dv ? *reinterpret_cast<const float2*>(vals + (jj + e) * Dv + 64 * i) : make_float2(0.f, 0.f);
#pragma unroll
                        for (int r = 0; r < R; ++r) {
                            const float4 p4 = *reinterpret_cast<const float4*>(sp + r * TF_KEYS + jj);
                            const float pe[4] = {p4.x, p4.y, p4.z, p4.w};
                            const unsigned s4 = seen[r] >> jj;
#pragma unroll
                            for (int e = 0; e < 4; ++e)
#pragma unroll
                                for (int i = 0; i < VP; ++i) {
                                    const float a = fmaf(pe[e], v[e][i].x, acc[r][i][0]), b = fmaf(pe[e], v[e][i].y, acc[r][i][1]);
                                    acc[r][i][0] = s4 & (1u << e) ? a : acc[r][i][0];
                                    acc[r][i][1] = s4 & (1u << e) ? b : acc[r][i][1];
                                }
                        }
                    }
                }
#pragma unroll
                for (int r = 0; r < R; ++r)
#pragma unroll
                    for (int i = 0; i < VP; ++i)
                        if (2 * lane + 64 * i < Dv) *reinterpret_cast<float2*>(mine + r * SP + 2 * lane + 64 * i) = make_float2(acc[r][i][0], acc[r][i][1]);
                visited |= 1u << cls;
                __syncwarp();
            }
            __syncthreads();                               // the buffer may be filled again
        }
        asm volatile("cp.async.wait_group 0;\n" ::);
        // the classes of the warp's rows meet, in their order
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int t = warp * R + r;
            if (t < start || t >= end) continue;
            float top = -INFINITY, L = 0.f, o[VP][2];
#pragma unroll
            for (int i = 0; i < VP; ++i) o[i][0] = o[i][1] = 0.f;
            for (int w = 0; w < TF_CLASSES; ++w)
                if (visited >> w & 1u) top = fmaxf(top, state[(size_t)(w * R + r) * SP + Dv]);
            for (int w = 0; w < TF_CLASSES; ++w) {
                if (!(visited >> w & 1u)) continue;
                const float* src = state + (size_t)(w * R + r) * SP;
                const float f = src[Dv] == -INFINITY ? 0.f : expf(src[Dv] - top);
                L = fmaf(src[Dv + 1], f, L);
#pragma unroll
                for (int i = 0; i < VP; ++i)
                    if (2 * lane + 64 * i < Dv) {
                        const float2 a = *reinterpret_cast<const float2*>(src + 2 * lane + 64 * i);
                        o[i][0] = fmaf(a.x, f, o[i][0]); o[i][1] = fmaf(a.y, f, o[i][1]);
                    }
            }
            float keep = 1.f;
            if (sink) {                                    // one more term of the denominator: exp(sink), with no key and no value
                const float all = fmaxf(top, sink[h]);
                keep = expf(top - all);
                L = L * keep + expf(sink[h] - all);
            }
            const float f = keep / L;
            float* dst = out + ((size_t)(t0 + t) * H + h) * Dv;
#pragma unroll
            for (int i = 0; i < VP; ++i)
                if (2 * lane + 64 * i < Dv) { dst[2 * lane + 64 * i] = o[i][0] * f; dst[2 * lane + 64 * i + 1] = o[i][1] * f; }
        }
        __syncthreads();                                   // (the next turn's chunks take the buffers)
        start = end;
    }
}

template <int R, int VP>
int launch_tiles(const float* q, int q_row_stride, const float* kpages, const float* vpages, const int* block_table, int max_blocks, const int* positions,
                 const int* seq_of_token, const float* rel, const int* bucket_of, int far, float* out, int n_tokens, int H, int Hkv, int Dk, int Dv, float scale,
                 int window, int keep_first, int chunk, int n_pages, const float* sink, const float* slopes, int v_stride, int* err, cudaStream_t stream) {
    static VmOncePerDevice once;
    const cudaError_t e = vm_allow_smem(once, attn_tiles_f32_kernel<R, VP>, TF_MOST_BYTES);
    if (e != cudaSuccess) return (int)e;
    const dim3 grid((n_tokens + TF_WARPS * R - 1) / (TF_WARPS * R), H);
    attn_tiles_f32_kernel<R, VP><<<grid, TF_WARPS * 32, tf_bytes(R, Dk, Dv, tf_classes(max_blocks)), stream>>>(
        q, q_row_stride, kpages, vpages, block_table, max_blocks, positions, seq_of_token, rel, bucket_of, far, out, n_tokens, H, Hkv, Dk, Dv, scale, window,
        keep_first, chunk, n_pages, sink, slopes, v_stride, err);
    return vm_launch_status();
}

}  // namespace

// 1 if vm_attention_tiles_f32 takes these sizes (16-byte pieces of keys and values; what it keeps of a tile fits shared memory)
VM_API int vm_attention_tiles_f32_fits(const void* kpages, const void* vpages, int H, int Dk, int Dv, int v_stride) {
    return Dk % 4 == 0 && Dk <= 256 && Dv % 4 == 0 && Dv <= 128 && v_stride % 4 == 0 && H <= 65535 && reinterpret_cast<uintptr_t>(kpages) % 16 == 0 &&
                   reinterpret_cast<uintptr_t>(vpages) % 16 == 0 && tf_bytes(4, Dk, Dv, TF_CLASSES) <= TF_MOST_BYTES
               ? 1
               : 0;
}

// arguments as vm_attention_rows in float32; rows_per_warp: 2, 4 or 8 (any gives the same result), 0: by the step's shape
VM_API int vm_attention_tiles_f32(const void* q, int q_row_stride, const void* kpages, const void* vpages, const int* block_table, int max_blocks,
                                  const int* positions, const int* seq_of_token, const float* rel, const int* bucket_of, int far, const float* sink,
                                  const float* slopes, int v_stride, void* out, int n_tokens, int H, int Hkv, int Dk, int Dv, float scale, int window,
                                  int keep_first, int chunk, int n_pages, int* err, int rows_per_warp, cudaStream_t stream) {
    if (n_tokens <= 0) return 0;
    if (!vm_attention_tiles_f32_fits(kpages, vpages, H, Dk, Dv, v_stride)) return VM_ERR_UNSUPPORTED;
    // Rows of a warp: the most that leave two CTAs for every SM and two of them room on it (four prompts of 33 to 190 tokens, 9 heads: 24.7 / 31 / 43 us with 2 / 4 / 8 rows;
    // one of 2,048 tokens 524 / 470 / 543)
    int R = rows_per_warp;
    if (R == 0)
        for (R = 8; R > 2; R /= 2)
            if (tf_bytes(R, Dk, Dv, tf_classes(max_blocks)) <= 110 * 1024 && (long long)(n_tokens + 4 * R - 1) / (4 * R) * H >= 2ll * vm_sm_count()) break;
#define VM_TILES(RR, P)                                                                                                                                    \
    if (R == RR && Dv <= 64 * P)                                                                                                                           \
        return launch_tiles<RR, P>((const float*)q, q_row_stride, (const float*)kpages, (const float*)vpages, block_table, max_blocks, positions,          \
                                   seq_of_token, rel, bucket_of, far, (float*)out, n_tokens, H, Hkv, Dk, Dv, scale, window, keep_first, chunk, n_pages, sink, \
                                   slopes, v_stride, err, stream);
    if (tf_bytes(R, Dk, Dv, tf_classes(max_blocks)) <= TF_MOST_BYTES) { VM_TILES(2, 1) VM_TILES(2, 2) VM_TILES(4, 1) VM_TILES(4, 2) VM_TILES(8, 1) VM_TILES(8, 2) }
#undef VM_TILES
    return VM_ERR_UNSUPPORTED;
}
