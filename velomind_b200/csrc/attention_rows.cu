// Attention over the paged cache in float32 arithmetic with the work of a query spread over a CTA: the kernel of the true 32-bit path
// (and of bfloat16 shapes that the tensor-core kernels refuse) for head sizes in multiples of four.  Options as in attention_biased.cu:
// a bias by bucketed distance, slopes, a sink, a window with kept first tokens, a chunked mask, values inside the key rows.
//
// What bounds it is latency: a decode step of a few sequences is a chain of loads.  With one warp per (token, head) that chain was as
// long as the context (120 us for four tokens of 9 heads at 190 cached tokens, 122 us for 446 tokens of four prompts).  Here a CTA owns up to
// eight query rows that share a kv head (the heads of its group, of one or more neighbouring tokens), and its eight warps share the
// keys: a chunk of 32 keys, one key per lane, belongs to the warp with its number modulo eight (a table of one or two pages has two or four chunks, and
// the CTA as many warps).  The key rows come as whole lines, all in
// flight, and pass through the warp's own shared memory (a lane that reads its row from global memory touches a line of its own with every
// load: 5 us a chunk instead of 2); a value row is one line; the probabilities come from shared memory four at a time; the warps' sums meet
// in warp order at the end.
// Measured at those sizes: 6.2 us and 59 us; one prompt of 8, 190, 446 and 2,048 tokens 4.7, 24, 75 and 800 us (5.7, 90, 322 and 5,049 before).  Where there
// are hardly any keys the join costs more than it saves: a first token alone 4.3 us (3.9 before), sixteen prompts of 8 tokens and 9 heads 8.5 (6.8).
//
// The result for a query depends on its own place alone: chunks start at absolute multiples of 32, which warp takes one follows from its
// absolute number, every dot product is summed in index order by one lane, and the other rows of a CTA never enter a row's arithmetic.
// So it does not matter how tokens were cut into steps, what else is in the batch, or how many rows a CTA was given.
#include "common.cuh"

namespace {

constexpr int MAX_ROWS = 8;
// Prompts that take attention_tiles_f32.cu: eight tokens a sequence and more, enough rows to fill the GPU, no long cached prefix (whose keys the warps here share)
bool tiles_pay(int n_tokens, int n_seqs, int H, int max_blocks) {
    return n_seqs > 0 && n_tokens >= 8 * n_seqs && (long long)n_tokens * H >= 2000 && (max_blocks == 1 || 16ll * max_blocks * n_seqs <= n_tokens);
}
constexpr int KEYS = 32;                 // keys of a warp's turn
constexpr int SLICE = 64;                // columns of the keys in shared memory at a time
template <typename T> constexpr int pitch() { return SLICE + 16 / (int)sizeof(T); }      // of a key row there: a lane's row starts 16 bytes further round the banks
template <typename T> struct four_of { using type = float4; };
template <> struct four_of<__nv_bfloat16> { using type = uint2; };

// four neighbouring values of a row (Dk is a multiple of 4, so 16- or 8-byte aligned)
__device__ __forceinline__ float4 load4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 load4(const __nv_bfloat16* p) {
    const uint2 u = *reinterpret_cast<const uint2*>(p);
    const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.x)), b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.y));
    return make_float4(a.x, a.y, b.x, b.y);
}
__device__ __forceinline__ float2 load2(const float* p) { return *reinterpret_cast<const float2*>(p); }
__device__ __forceinline__ float2 load2(const __nv_bfloat16* p) { return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(p)); }

// R: query rows of a CTA (a power of two); VP: pairs of value columns per lane, 2 lane + 64 i and the next; WARPS: 8, or as many as the table has chunks
template <typename T, int R, int VP, int WARPS>
__global__ void __launch_bounds__(WARPS * 32)
attn_rows_kernel(const T* __restrict__ q, int q_row_stride, const T* __restrict__ kpages, const T* __restrict__ vpages,
                 const int* __restrict__ block_table, int max_blocks, const int* __restrict__ positions, const int* __restrict__ seq_of_token,
                 const float* __restrict__ rel, const int* __restrict__ bucket_of, int far, T* __restrict__ out, int n_tokens, int tile_tokens,
                 int H, int Hkv, int Dk, int Dv, float scale, int window, int keep_first, int chunk, int n_pages, const float* __restrict__ sink,
                 const float* __restrict__ slopes, int v_stride, int* __restrict__ err) {
    extern __shared__ __align__(16) float sm[];
    float* sq = sm;                                        // [R][Dk] scaled queries
    float* sp = sq + R * Dk;                               // [WARPS][R][32] probabilities of a warp's chunk
    float* part = sp + WARPS * R * 32;                     // [WARPS][R][Dv + 2] sums, then maximum and denominator, behind the keys
    using Unit = typename four_of<T>::type;
    constexpr int PITCH = pitch<T>();
    T* keys = reinterpret_cast<T*>(part) + (threadIdx.x >> 5) * KEYS * PITCH;      // [WARPS][KEYS][PITCH]: a warp's slice of its keys (the sums take their place at the end)
    const int G = H / Hkv, groups = (G + R - 1) / R;
    const int hk = blockIdx.y / groups, h0 = hk * G + (blockIdx.y - hk * groups) * R;
    const int heads = min(R, hk * G + G - h0);             // query heads of this CTA; row r is token r / heads, head r % heads
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int t_end = min(n_tokens, (int)(blockIdx.x + 1) * tile_tokens);

    for (int t0 = blockIdx.x * tile_tokens; t0 < t_end;) {
        // the neighbouring tokens of one sequence (a tile may cross into the next one: another turn)
        const int seq = seq_of_token[t0];
        int t1 = t0 + 1;
        while (t1 < t_end && seq_of_token[t1] == seq) ++t1;
        const int rows = (t1 - t0) * heads;
        int pos[R], lo[R], head[R], lowest = 0x7fffffff, highest = -1, kept_most = 0;
#pragma unroll
        for (int r = 0, t = t0, h = h0; r < R; ++r) {
            pos[r] = -1; lo[r] = 0x7fffffff;               // a row that is not there sees nothing
            head[r] = h;
            if (r < rows) {
                pos[r] = positions[t];
                lo[r] = vm_first_seen(pos[r], window, chunk);
                lowest = min(lowest, lo[r]);
                highest = max(highest, pos[r]);
                kept_most = max(kept_most, min(keep_first, lo[r]));
            }
            if (++h == h0 + heads) { h = h0; ++t; }
        }
        // this warp's first chunk (not between the kept tokens and the window) and its page, asked for before the queries' barrier
        auto next_chunk = [&](int c) {
            if (c * 32 >= kept_most && c < lowest / 32) c += (lowest / 32 - c + WARPS - 1) / WARPS * WARPS;
            return c;
        };
        auto page_of = [&](int c) {
            const int blk = c * 32 / VM_PAGE_TOKENS;
            return c * 32 <= highest && blk < max_blocks ? block_table[(size_t)seq * max_blocks + blk] : -1;
        };
        int c = next_chunk(warp), page = page_of(c);
        const int first = c * 32;
        for (int i = threadIdx.x; i < R * Dk; i += WARPS * 32) {
            const int r = i / Dk, d = i - r * Dk;
            sq[i] = r < rows ? vm_to_float(q[(size_t)(t0 + r / heads) * q_row_stride + (size_t)(h0 + r % heads) * Dk + d]) * scale : 0.f;
        }
        __syncthreads();
        float m[R], l[R], acc[R][VP][2];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            m[r] = -INFINITY; l[r] = 0.f;
#pragma unroll
            for (int i = 0; i < VP; ++i) acc[r][i][0] = acc[r][i][1] = 0.f;
        }
        float* mine = sp + warp * R * 32;
        for (; c * 32 <= highest; c = next_chunk(c + WARPS)) {
            const int base = c * 32;
            if (base != first) page = page_of(c);
            if (page < 0 || page >= n_pages) {             // a page the step needs is not there: report, skip
                if (lane == 0 && err) atomicExch(err, VM_ERRWORD_CACHE_READ);
                continue;
            }
            const size_t tok0 = ((size_t)page * Hkv + hk) * VM_PAGE_TOKENS + (base % VM_PAGE_TOKENS);
            const int j = base + lane;
            const T* vrow = vpages + tok0 * v_stride + 2 * lane;
            const int last = min(KEYS - 1, highest - base);
            float s[R];
#pragma unroll
            for (int r = 0; r < R; ++r) s[r] = 0.f;
            // 64 columns of the 32 key rows at a time: fetched as whole lines, kept in the warp's own shared memory, read back a row per lane
            const int rows_here = min(KEYS, highest - base + 1);
            for (int d0 = 0; d0 < Dk; d0 += SLICE) {
                const int units = min(SLICE, Dk - d0) / 4;                 // of four values
                const T* src = kpages + tok0 * Dk + d0;
                if (units == SLICE / 4) {
                    Unit got[KEYS * SLICE / 4 / 32];
#pragma unroll
                    for (int k = 0; k < KEYS * SLICE / 4 / 32; ++k) {
                        const int u = lane + 32 * k, row = u / (SLICE / 4), col = u % (SLICE / 4);
                        if (row < rows_here) got[k] = *reinterpret_cast<const Unit*>(src + (size_t)row * Dk + 4 * col);
                    }
#pragma unroll
                    for (int k = 0; k < KEYS * SLICE / 4 / 32; ++k) {
                        const int u = lane + 32 * k, row = u / (SLICE / 4), col = u % (SLICE / 4);
                        if (row < rows_here) *reinterpret_cast<Unit*>(keys + row * PITCH + 4 * col) = got[k];
                    }
                } else {
                    for (int u = lane; u < rows_here * units; u += 32) {
                        const int row = u / units, col = u - row * units;
                        *reinterpret_cast<Unit*>(keys + row * PITCH + 4 * col) = *reinterpret_cast<const Unit*>(src + (size_t)row * Dk + 4 * col);
                    }
                }
                __syncwarp();
                if (j <= highest) {
#pragma unroll 4
                    for (int d = 0; d < 4 * units; d += 4) {
                        const float4 k4 = load4(keys + lane * PITCH + d);
#pragma unroll
                        for (int r = 0; r < R; ++r) {
                            const float4 q4 = *reinterpret_cast<const float4*>(sq + r * Dk + d0 + d);
                            s[r] = fmaf(q4.x, k4.x, s[r]); s[r] = fmaf(q4.y, k4.y, s[r]);
                            s[r] = fmaf(q4.z, k4.z, s[r]); s[r] = fmaf(q4.w, k4.w, s[r]);
                        }
                    }
                }
                __syncwarp();
            }
            // the first value rows are on their way while the scores become probabilities
            auto load_values = [&](int jj, float2 (&v)[4][VP]) {
#pragma unroll
                for (int e = 0; e < 4; ++e)
#pragma unroll
                    for (int i = 0; i < VP; ++i)
                        v[e][i] = 2 * lane + 64 * i < Dv ? load2(vrow + (size_t)min(jj + e, last) * v_stride + 64 * i) : make_float2(0.f, 0.f);
            };
            constexpr int EARLY = 8 / VP;                  // groups of four rows
            float2 early[EARLY][4][VP];
#pragma unroll
            for (int k = 0; k < EARLY; ++k) load_values(4 * k, early[k]);
            unsigned seen[R];                              // which of the chunk's keys each row sees
            bool all_seen = true;
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const bool valid = j <= pos[r] && (j >= lo[r] || j < min(keep_first, lo[r]));
                seen[r] = __ballot_sync(0xffffffffu, valid);
                all_seen = all_seen && (r >= rows || seen[r] == 0xffffffffu);
                float x = -INFINITY;
                if (valid) {
                    x = s[r];
                    if (rel) x += rel[(size_t)bucket_of[min(pos[r] - j, far)] * H + head[r]];
                    if (slopes) x = fmaf(-slopes[head[r]], (float)(pos[r] - j), x);
                }
                const float top = fmaxf(m[r], vm_warp_max(x));
                const float use = top == -INFINITY ? 0.f : top;      // nothing seen so far: no factor changes anything
                const float p = valid ? expf(x - use) : 0.f;
                const float alpha = expf(m[r] - use);
                l[r] = fmaf(l[r], alpha, vm_warp_sum(p));
#pragma unroll
                for (int i = 0; i < VP; ++i) { acc[r][i][0] *= alpha; acc[r][i][1] *= alpha; }
                m[r] = top;
                mine[r * 32 + lane] = p;
            }
            __syncwarp();
            // values of 32 keys; at the edge of a mask a row takes the ones it sees and no others (they may hold anything, infinities too)
            if (all_seen) {
                auto add = [&](int jj, const float2 (&v)[4][VP]) {
#pragma unroll
                    for (int r = 0; r < R; ++r) {
                        const float4 p4 = *reinterpret_cast<const float4*>(mine + r * 32 + jj);
                        const float pe[4] = {p4.x, p4.y, p4.z, p4.w};
#pragma unroll
                        for (int e = 0; e < 4; ++e)
#pragma unroll
                            for (int i = 0; i < VP; ++i) {
                                acc[r][i][0] = fmaf(pe[e], v[e][i].x, acc[r][i][0]);
                                acc[r][i][1] = fmaf(pe[e], v[e][i].y, acc[r][i][1]);
                            }
                    }
                };
#pragma unroll
                for (int k = 0; k < EARLY; ++k) add(4 * k, early[k]);
#pragma unroll
                for (int k = EARLY; k < KEYS / 4; ++k) {
                    float2 v[4][VP];
                    load_values(4 * k, v);
                    add(4 * k, v);
                }
            } else {
                auto add = [&](int jj, const float2 (&v)[4][VP]) {
#pragma unroll
                    for (int r = 0; r < R; ++r) {
                        const float4 p4 = *reinterpret_cast<const float4*>(mine + r * 32 + jj);
                        const float pe[4] = {p4.x, p4.y, p4.z, p4.w};
                        const unsigned s4 = seen[r] >> jj;
#pragma unroll
                        for (int e = 0; e < 4; ++e)
#pragma unroll
                            for (int i = 0; i < VP; ++i) {
                                const float x = fmaf(pe[e], v[e][i].x, acc[r][i][0]), y = fmaf(pe[e], v[e][i].y, acc[r][i][1]);
                                acc[r][i][0] = s4 & (1u << e) ? x : acc[r][i][0];
                                acc[r][i][1] = s4 & (1u << e) ? y : acc[r][i][1];
                            }
                    }
                };
#pragma unroll
                for (int k = 0; k < EARLY; ++k)
                    if (4 * k <= last) add(4 * k, early[k]);
#pragma unroll
                for (int k = EARLY; k < KEYS / 4; ++k) {
                    if (4 * k > last) break;
                    float2 v[4][VP];
                    load_values(4 * k, v);
                    add(4 * k, v);
                }
            }
            __syncwarp();                                  // the next chunk's probabilities take this one's place
        }
        __syncthreads();                                   // (no warp reads keys any more)
#pragma unroll
        for (int r = 0; r < R; ++r) {
            float* dst = part + (size_t)(warp * R + r) * (Dv + 2);
            if (lane == 0) { dst[Dv] = m[r]; dst[Dv + 1] = l[r]; }
#pragma unroll
            for (int i = 0; i < VP; ++i) {
                const int d = 2 * lane + 64 * i;
                if (d < Dv) { dst[d] = acc[r][i][0]; dst[d + 1] = acc[r][i][1]; }
            }
        }
        __syncthreads();
        for (int i = threadIdx.x; i < rows * Dv; i += WARPS * 32) {
            const int r = i / Dv, d = i - r * Dv, h = h0 + r % heads;
            const float* src = part + (size_t)r * (Dv + 2);
            const size_t step = (size_t)R * (Dv + 2);
            float top = -INFINITY;
#pragma unroll
            for (int w = 0; w < WARPS; ++w) top = fmaxf(top, src[w * step + Dv]);
            float o = 0.f, L = 0.f;
#pragma unroll
            for (int w = 0; w < WARPS; ++w) {              // in warp order: the same sum whatever else runs
                const float f = src[w * step + Dv] == -INFINITY ? 0.f : expf(src[w * step + Dv] - top);
                o = fmaf(src[w * step + d], f, o);
                L = fmaf(src[w * step + Dv + 1], f, L);
            }
            float keep = 1.f;
            if (sink) {                                    // one more term of the denominator: exp(sink), with no key and no value
                const float all = fmaxf(top, sink[h]);
                keep = expf(top - all);
                L = L * keep + expf(sink[h] - all);
            }
            out[((size_t)(t0 + r / heads) * H + h) * Dv + d] = vm_from_float<T>(o * (keep / L));
        }
        __syncthreads();
        t0 = t1;
    }
}

template <typename T, int R, int VP, int WARPS>
int launch_rows(const void* q, int q_row_stride, const void* kpages, const void* vpages, const int* block_table, int max_blocks, const int* positions,
                const int* seq_of_token, const float* rel, const int* bucket_of, int far, void* out, int n_tokens, int tile_tokens, int H, int Hkv,
                int Dk, int Dv, float scale, int window, int keep_first, int chunk, int n_pages, const float* sink, const float* slopes, int v_stride,
                int* err, cudaStream_t stream) {
    const size_t keys = (size_t)WARPS * KEYS * pitch<T>() * sizeof(T), sums = (size_t)WARPS * R * (Dv + 2) * sizeof(float);
    const size_t smem = ((size_t)R * Dk + (size_t)WARPS * R * 32) * sizeof(float) + (keys > sums ? keys : sums);
    static VmOncePerDevice once;
    const cudaError_t e = vm_allow_smem(once, attn_rows_kernel<T, R, VP, WARPS>, 100 * 1024);
    if (e != cudaSuccess) return (int)e;
    const int G = H / Hkv;
    const dim3 grid((n_tokens + tile_tokens - 1) / tile_tokens, Hkv * ((G + R - 1) / R));
    attn_rows_kernel<T, R, VP, WARPS><<<grid, WARPS * 32, smem, stream>>>((const T*)q, q_row_stride, (const T*)kpages, (const T*)vpages, block_table, max_blocks,
                                                                   positions, seq_of_token, rel, bucket_of, far, (T*)out, n_tokens, tile_tokens, H, Hkv,
                                                                   Dk, Dv, scale, window, keep_first, chunk, n_pages, sink, slopes, v_stride, err);
    return vm_launch_status();
}

template <typename T>
int dispatch_rows(const void* q, int q_row_stride, const void* kpages, const void* vpages, const int* block_table, int max_blocks, const int* positions,
                  const int* seq_of_token, const float* rel, const int* bucket_of, int far, void* out, int n_tokens, int H, int Hkv, int Dk, int Dv,
                  float scale, int window, int keep_first, int chunk, int n_pages, const float* sink, const float* slopes, int v_stride, int* err,
                  int n_seqs, cudaStream_t stream) {
    // None of what is chosen here changes a row's result, so all of it may follow from the step's shape.
    // Warps: eight, or a table's two or four chunks of keys and no more: 64 tokens or fewer leave two warps with work, and the CTAs are smaller (30 tokens
    // of 9 heads 5.4 us with two warps, 8.2 with eight; 16 sequences of 60 tokens, 32 heads 6.2 / 19.7).
    // Rows: as few as keep the CTAs within what the SMs hold side by side (a CTA's chain grows with its rows: one sequence of 190 tokens and
    // 9 heads 6.4 / 7.2 / 8.9 us with 1 / 2 / 4 rows), then as many as a kv head has, up to eight (64 sequences of 500 tokens and 9 heads 26.7 us
    // with 4 rows, 29.7 with 2, 34.4 with 1; a prompt of 446 tokens 75 us with 8, 158 with 1).
    // Neighbouring tokens share a CTA only as far as sequences bring several: those of different sequences are taken one after another (16 sequences of 190
    // tokens, 32 heads without groups: 21.7 us a CTA per token, 81 us with eight tokens in a CTA).
    const int G = H / Hkv, warps = max_blocks <= 1 ? 2 : max_blocks <= 2 ? 4 : 8;
    const int together = n_seqs > 0 ? (n_tokens / n_seqs > 1 ? n_tokens / n_seqs : 1) : n_tokens;
    const long long room = (long long)vm_sm_count() * 8 / warps;
    int R = 1, tile = 1;
    for (;; R *= 2) {
        tile = R / G < 1 ? 1 : R / G < together ? R / G : together;
        if (R == MAX_ROWS || R >= (long long)G * together || (n_tokens + tile - 1ll) / tile * Hkv * ((G + R - 1) / R) <= room) break;
    }
    const int vp = (Dv + 63) / 64;
#define VM_ROWS_WARPS(RR, P, W)                                                                                                                 \
    if (R == RR && vp <= P && warps == W)                                                                                                       \
        return launch_rows<T, RR, P, W>(q, q_row_stride, kpages, vpages, block_table, max_blocks, positions, seq_of_token, rel, bucket_of, far, out, \
                                        n_tokens, tile, H, Hkv, Dk, Dv, scale, window, keep_first, chunk, n_pages, sink, slopes, v_stride, err, stream);
#define VM_ROWS(RR, P) VM_ROWS_WARPS(RR, P, 2) VM_ROWS_WARPS(RR, P, 4) VM_ROWS_WARPS(RR, P, 8)
    VM_ROWS(1, 1) VM_ROWS(2, 1) VM_ROWS(4, 1) VM_ROWS(8, 1)
    VM_ROWS(1, 2) VM_ROWS(2, 2) VM_ROWS(4, 2) VM_ROWS(8, 2)
#undef VM_ROWS
#undef VM_ROWS_WARPS
    return VM_ERR_UNSUPPORTED;
}

}  // namespace

// 1 if vm_attention_rows takes these sizes and rows (16-byte loads of keys, pairs of values; what it keeps of eight rows fits shared memory)
VM_API int vm_attention_rows_fits(const void* kpages, const void* vpages, int H, int Hkv, int Dk, int Dv, int v_stride) {
    return Dk % 4 == 0 && Dk <= 512 && Dv % 2 == 0 && Dv <= 128 && v_stride % 2 == 0 && reinterpret_cast<uintptr_t>(kpages) % 16 == 0 &&
                   reinterpret_cast<uintptr_t>(vpages) % 8 == 0 && (long long)Hkv * ((H / Hkv + MAX_ROWS - 1) / MAX_ROWS) <= 65535
               ? 1
               : 0;
}

// n_seqs: sequences of the step (0: not known, its tokens are taken for a prompt's)
VM_API int vm_attention_rows(const void* q, int q_row_stride, const void* kpages, const void* vpages, const int* block_table, int max_blocks,
                             const int* positions, const int* seq_of_token, const float* rel, const int* bucket_of, int far, const float* sink,
                             const float* slopes, int v_stride, void* out, int n_tokens, int H, int Hkv, int Dk, int Dv, float scale, int window,
                             int keep_first, int chunk, int n_pages, int act_dtype, int* err, int n_seqs, cudaStream_t stream) {
    if (n_tokens <= 0) return 0;
    if (!vm_attention_rows_fits(kpages, vpages, H, Hkv, Dk, Dv, v_stride)) return VM_ERR_UNSUPPORTED;
    if (act_dtype == VM_F32 && tiles_pay(n_tokens, n_seqs, H, max_blocks) && vm_attention_tiles_f32_fits(kpages, vpages, H, Dk, Dv, v_stride))
        return vm_attention_tiles_f32(q, q_row_stride, kpages, vpages, block_table, max_blocks, positions, seq_of_token, rel, bucket_of, far, sink, slopes,
                                      v_stride, out, n_tokens, H, Hkv, Dk, Dv, scale, window, keep_first, chunk, n_pages, err, 0, stream);
    if (act_dtype == VM_F32)
        return dispatch_rows<float>(q, q_row_stride, kpages, vpages, block_table, max_blocks, positions, seq_of_token, rel, bucket_of, far, out, n_tokens, H,
                                    Hkv, Dk, Dv, scale, window, keep_first, chunk, n_pages, sink, slopes, v_stride, err, n_seqs, stream);
    if (act_dtype == VM_BF16)
        return dispatch_rows<__nv_bfloat16>(q, q_row_stride, kpages, vpages, block_table, max_blocks, positions, seq_of_token, rel, bucket_of, far, out,
                                            n_tokens, H, Hkv, Dk, Dv, scale, window, keep_first, chunk, n_pages, sink, slopes, v_stride, err, n_seqs, stream);
    return VM_ERR_UNSUPPORTED;
}
