// Products of a few rows (M <= 32, decode steps) in bfloat16 whose rows lie READY in memory: plain bfloat16 rows, or rows of the residual stream that
// the kernel in front left as x times the coming norm's weight, with the parts of their sums of squares beside them.
//
// Bound by latency: 0.6 to 4 MB of weights a launch, and a chain of launches of which each needs the one before.  An empty launch of such a chain under
// programmatic dependent launch takes 0.5 us, one that reads a row and writes 1.0 us; everything above that is this kernel's own chain.  The kernel of
// skinny_body.cuh copies the rows (of a norm: the float32 stream, with the squares summed and the values converted by EVERY block) into shared memory and
// meets there before it multiplies.  Here nothing is staged: a lane's 16 bytes of a weight row are the A fragments of two mma.sync m16n8k16 (k permuted
// alike in both operands), its 16 bytes of an activation row the B fragments, both straight from global memory; weights are requested before the wait on
// the kernel in front, rows after it, and the warps (which share K) meet once, over the sums.  A warp of its own joins the sums of squares meanwhile: done
// by the multiplying warps in front of their products it cost 0.5 us.
//
// The residual epilogue leaves the new rows ready for the next product: ready = bf16(h x next norm's weight) and, per row and block, the sum of squares of
// the h just written (float32, joined by the reader in a fixed order).
//
// Measured in a chain of launches under a graph (weights from DRAM), old kernel -> this one, 1 and 8 rows: 960 x 576 with norm, rotation and cache write
// 3.15 -> 1.9, 3.3 -> 2.0 us; 576 x 576 with the residual sum 2.3 -> 1.5, 2.45 -> 1.65; 2 x 1,536 x 576 with norm and unit 3.2 -> 2.0, 3.45 -> 2.3;
// 576 x 1,536 with the sum 3.2 -> 1.7, 3.3 -> 1.9.  Larger matrices, against the kernel of skinny_stream.cuh, 8 rows: 960 x 2,560 5.4 -> 2.7,
// 2 x 2,560 x 960 5.9 -> 3.4, 2,048 x 8,192 11.8 -> 8.2 (33.6 MB: 4.1 TB/s), 6,144 x 2,048 7.9 -> 5.9, 2 x 8,192 x 2,048 14.7 -> 13.8 (4.9 TB/s).
// 17 and 32 plain rows: 960 x 576 3.4 -> 2.0, 3.8 -> 2.2; 2 x 1,536 x 576 4.35 -> 3.6, 5.0 -> 3.8; 576 x 1,536 with the sum 3.3 -> 3.0, 3.6 -> 3.3; 2 x 2,560 x 960
// 7.9 -> 7.5, 9.9 -> 8.1; 960 x 2,560 with the sum 6.0 -> 5.5, 7.1 -> 5.9; 2,048 x 2,048 with the sum 10.4 -> 4.7, 11.9 -> 5.2.  Where it loses, plain rows do not
// take it (ring_pays in skinny_gemm.cu).
#include "skinny_body.cuh"

namespace {

using namespace vmsk;

enum { DIRECT_STORE = 0, DIRECT_RESIDUAL = 1, DIRECT_UNIT = 2, DIRECT_ROPE = 3 };

__device__ __forceinline__ uint4 from_l2(const void* p) { return __ldcg(reinterpret_cast<const uint4*>(p)); }   // (written by other SMs: past L1)

// NT: tiles of eight rows; WARPS share K, each with PF blocks of 32 values in flight; TP: pairs of column tiles (8 + 8 columns) a block takes.
// With `squares` the block has one warp more.
template <int NT, int PF, int WARPS, int TP, int EPI>
__global__ void __launch_bounds__(WARPS * 32 + 32, WARPS == 8 && NT == 1 ? 2 : 1)
skinny_direct_kernel(const SkinnyParams p) {
    constexpr int THREADS = WARPS * 32;
    constexpr int RS = 8 * NT + (NT == 1 ? 0 : 4);       // row of the partial sums: lanes of eight columns by four rows meet 32 banks
    constexpr int CELLS = 64 * NT * TP, TURNS = (CELLS + THREADS - 1) / THREADS;
    __shared__ float red[WARPS][TP * 16][RS];
    __shared__ float scale[8 * NT];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t4 = lane & 3;
    vm_pdl_launch_dependents();                          // (of the form that writes the cache too: its reader asks for the new row after its own wait, common.cuh)
    const bool two = EPI == DIRECT_UNIT || EPI == DIRECT_ROPE || p.tiles == 2;
    const int pairs = p.N / (two ? 16 : 8);
    int nA[TP], nB[TP], head[TP];
#pragma unroll
    for (int t = 0; t < TP; ++t) {                       // (past the last pair: the last one once more, not stored)
        const int item = min((int)blockIdx.x * TP + t, pairs - 1);
        head[t] = 0;
        if (EPI == DIRECT_UNIT) { nA[t] = 8 * item; nB[t] = p.I + nA[t]; }
        else if (EPI == DIRECT_ROPE) { const SkinnyCols c = skinny_cols(p, item); nA[t] = c.nA; nB[t] = c.nB; head[t] = c.head; }
        else if (two) { nA[t] = 16 * item; nB[t] = nA[t] + 8; }
        else nA[t] = nB[t] = 8 * item;
    }
    const int blocks = p.K / 32;
    const bool multiplies = EPI == DIRECT_RESIDUAL || warp < WARPS;      // (a residual product's rows are plain)
    uint4 wa[TP][PF], wb[TP][PF];
    auto fetch_w = [&](int u, int b) {
#pragma unroll
        for (int t = 0; t < TP; ++t) {
            wa[t][u] = wb[t][u] = make_uint4(0u, 0u, 0u, 0u);
            if (b < blocks) {
                wa[t][u] = __ldg(reinterpret_cast<const uint4*>(p.W + (size_t)(nA[t] + g) * p.K + 8 * t4 + 32 * b));
                if (two) wb[t][u] = __ldg(reinterpret_cast<const uint4*>(p.W + (size_t)(nB[t] + g) * p.K + 8 * t4 + 32 * b));
            }
        }
    };
    if (multiplies) {
#pragma unroll
        for (int u = 0; u < PF; ++u) fetch_w(u, warp + WARPS * u);
    }
    // the cells of the result that this thread finishes: columns cA and cB of row er
    int er[TURNS], cA[TURNS], cB[TURNS], hd[TURNS], at[TURNS];
    float fa[TURNS], fb[TURNS];                          // constants of the columns: next norm's weights, or the rotary frequency
#pragma unroll
    for (int i = 0; i < TURNS; ++i) {
        const int e = tid + THREADS * i, t = TP == 1 ? 0 : (e >> 3) % TP, c = e & 7;
        er[i] = multiplies && e < CELLS && (int)blockIdx.x * TP + t < pairs ? (e >> 3) / TP : p.M;
        cA[i] = nA[0] + c; cB[i] = nB[0] + c; hd[i] = head[0]; at[i] = t * 16 + c;
        if (TP > 1 && t) { cA[i] = nA[TP - 1] + c; cB[i] = nB[TP - 1] + c; hd[i] = head[TP - 1]; }
        fa[i] = fb[i] = 0.f;
        if (er[i] < p.M) {
            if (EPI == DIRECT_ROPE && hd[i] < p.H + p.Hkv && p.rot_dim > 0) fa[i] = p.inv_freq[cA[i] - hd[i] * p.D];
            if (EPI == DIRECT_RESIDUAL && p.next_w) { fa[i] = p.next_w[cA[i]]; if (two) fb[i] = p.next_w[cB[i]]; }
        }
    }
    vm_pdl_wait();                                       // from here on: data written by earlier kernels

    uint4 x[PF][NT];
    auto fetch_x = [&](int u, int b) {
#pragma unroll
        for (int n = 0; n < NT; ++n) {
            x[u][n] = make_uint4(0u, 0u, 0u, 0u);
            if (b < blocks && 8 * n + g < p.M) x[u][n] = from_l2(static_cast<const __nv_bfloat16*>(p.A) + (size_t)(8 * n + g) * p.K + 8 * t4 + 32 * b);
        }
    };
    if (multiplies) {
#pragma unroll
        for (int u = 0; u < PF; ++u) fetch_x(u, warp + WARPS * u);
    }
    // what the epilogue needs per row is requested behind the rows
    float res_a[TURNS], res_b[TURNS];
    int pos[TURNS], page[TURNS];
#pragma unroll
    for (int i = 0; i < TURNS; ++i) {
        res_a[i] = res_b[i] = 0.f; pos[i] = 0; page[i] = -1;
        if (er[i] < p.M) {
            if (EPI == DIRECT_RESIDUAL) {
                res_a[i] = __ldcg(p.h + (size_t)er[i] * p.N + cA[i]);
                if (two) res_b[i] = __ldcg(p.h + (size_t)er[i] * p.N + cB[i]);
            }
            if (EPI == DIRECT_ROPE) {
                pos[i] = p.positions[er[i]];
                if (p.kpages != nullptr && hd[i] >= p.H) {
                    const int blk = pos[i] / VM_PAGE_TOKENS;
                    page[i] = (blk < p.max_blocks) ? p.block_table[(size_t)p.seq_of_token[er[i]] * p.max_blocks + blk] : -1;
                }
            }
        }
    }
    if (multiplies) {
        float acc[TP][NT][4];
#pragma unroll
        for (int t = 0; t < TP; ++t)
#pragma unroll
            for (int n = 0; n < NT; ++n) acc[t][n][0] = acc[t][n][1] = acc[t][n][2] = acc[t][n][3] = 0.f;
        for (int b0 = warp; b0 < blocks; b0 += WARPS * PF) {
            const bool more = b0 + WARPS * PF < blocks;
#pragma unroll
            for (int u = 0; u < PF; ++u) {
#pragma unroll
                for (int t = 0; t < TP; ++t)
#pragma unroll
                    for (int n = 0; n < NT; ++n) {
                        vm_mma_bf16_16816(acc[t][n], wa[t][u].x, wb[t][u].x, wa[t][u].y, wb[t][u].y, x[u][n].x, x[u][n].y);
                        vm_mma_bf16_16816(acc[t][n], wa[t][u].z, wb[t][u].z, wa[t][u].w, wb[t][u].w, x[u][n].z, x[u][n].w);
                    }
                if (more) { fetch_w(u, b0 + WARPS * (PF + u)); fetch_x(u, b0 + WARPS * (PF + u)); }
            }
        }
#pragma unroll
        for (int t = 0; t < TP; ++t)
#pragma unroll
            for (int n = 0; n < NT; ++n) {
                *reinterpret_cast<float2*>(&red[warp][t * 16 + g][8 * n + 2 * t4]) = make_float2(acc[t][n][0], acc[t][n][1]);
                if (two) *reinterpret_cast<float2*>(&red[warp][t * 16 + g + 8][8 * n + 2 * t4]) = make_float2(acc[t][n][2], acc[t][n][3]);
            }
    } else {
        // the rows' sums of squares: four lanes a row, all rows' parts in flight
        float s[NT];
#pragma unroll
        for (int n = 0; n < NT; ++n) s[n] = 0.f;
        const int quads = p.parts / 4;                   // (a row's parts are padded to whole float4)
        for (int i = t4; i < quads; i += 16) {
            float4 v[NT][4];
#pragma unroll
            for (int n = 0; n < NT; ++n)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    v[n][j] = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (8 * n + g < p.M && i + 4 * j < quads) v[n][j] = __ldcg(reinterpret_cast<const float4*>(p.squares + (size_t)(8 * n + g) * p.parts) + i + 4 * j);
                }
#pragma unroll
            for (int n = 0; n < NT; ++n)
#pragma unroll
                for (int j = 0; j < 4; ++j) s[n] += (v[n][j].x + v[n][j].y) + (v[n][j].z + v[n][j].w);
        }
#pragma unroll
        for (int n = 0; n < NT; ++n) {
            s[n] += __shfl_xor_sync(0xffffffffu, s[n], 1);
            s[n] += __shfl_xor_sync(0xffffffffu, s[n], 2);
            if (t4 == 0) scale[8 * n + g] = 1.0f / sqrtf(s[n] / (float)p.K + p.eps);
        }
    }
    if (EPI == DIRECT_ROPE) {                            // (cosine and sine take the constants' registers)
#pragma unroll
        for (int i = 0; i < TURNS; ++i)
            if (er[i] < p.M && hd[i] < p.H + p.Hkv && p.rot_dim > 0) sincosf((float)pos[i] * fa[i], &fb[i], &fa[i]);
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < TURNS; ++i) {
        const int row = er[i];
        if (row >= p.M) continue;                        // (whole groups of eight lanes leave together)
        float vA = 0.f, vB = 0.f;
#pragma unroll
        for (int w = 0; w < WARPS; ++w) {
            vA += red[w][at[i]][row];
            if (two) vB += red[w][at[i] + 8][row];
        }
        if (EPI != DIRECT_RESIDUAL && p.squares != nullptr) { const float rs = scale[row]; vA *= rs; vB *= rs; }
        if (EPI == DIRECT_STORE) {
            if (p.epi == EPI_STORE_F32) {
                float* o = static_cast<float*>(p.out) + (size_t)row * p.out_stride;
                o[cA[i]] = vA;
                if (two) o[cB[i]] = vB;
            } else {
                if (p.store_act) {       // the activation of what the product's bfloat16 result would hold, as the unfused step computes it
                    vA = skinny_gate(__bfloat162float(__float2bfloat16_rn(vA)), p.store_act - 1);
                    vB = skinny_gate(__bfloat162float(__float2bfloat16_rn(vB)), p.store_act - 1);
                }
                __nv_bfloat16* o = static_cast<__nv_bfloat16*>(p.out) + (size_t)row * p.out_stride;
                o[cA[i]] = __float2bfloat16_rn(vA);
                if (two) o[cB[i]] = __float2bfloat16_rn(vB);
            }
        } else if (EPI == DIRECT_RESIDUAL) {
            const float a = res_a[i] + vA, b = two ? res_b[i] + vB : 0.f;
            float* o = p.h + (size_t)row * p.N;
            o[cA[i]] = a;
            if (two) o[cB[i]] = b;
            if (p.next_w) {
                __nv_bfloat16* r = p.ready + (size_t)row * p.N;
                r[cA[i]] = __float2bfloat16_rn(a * fa[i]);
                if (two) r[cB[i]] = __float2bfloat16_rn(b * fb[i]);
                float s = a * a + b * b;
                const unsigned mask = 0xffu << (lane & 24);
                s += __shfl_xor_sync(mask, s, 1); s += __shfl_xor_sync(mask, s, 2); s += __shfl_xor_sync(mask, s, 4);
                float* sq = p.ready_squares + (size_t)row * p.ready_parts;
                if ((lane & 7) == 0) sq[blockIdx.x] = s;
                if (blockIdx.x == 0 && (lane & 7) && pairs + (lane & 7) - 1 < p.ready_parts) sq[pairs + (lane & 7) - 1] = 0.f;   // the padding
            }
        } else if (EPI == DIRECT_UNIT) {
            static_cast<__nv_bfloat16*>(p.out)[(size_t)row * p.out_stride + cA[i]] = __float2bfloat16_rn(skinny_unit(p, vA, vB));
        } else if (EPI == DIRECT_ROPE) {
            float ya = vA, yb = vB;
            if (hd[i] < p.H + p.Hkv && p.rot_dim > 0) { ya = vA * fa[i] - vB * fb[i]; yb = vB * fa[i] + vA * fb[i]; }
            const int da = cA[i] - hd[i] * p.D, db = cB[i] - hd[i] * p.D;
            if (hd[i] < p.H) {
                __nv_bfloat16* o = static_cast<__nv_bfloat16*>(p.out) + (size_t)row * p.out_stride + (size_t)hd[i] * p.D;
                o[da] = __float2bfloat16_rn(ya); o[db] = __float2bfloat16_rn(yb);
            } else if (p.kpages != nullptr) {
                if (page[i] < 0 || page[i] >= p.n_pages) { if (p.err) atomicExch(p.err, 2); continue; }
                const bool is_k = hd[i] < p.H + p.Hkv;
                const int hk = is_k ? hd[i] - p.H : hd[i] - p.H - p.Hkv;
                __nv_bfloat16* dst = (is_k ? p.kpages : p.vpages) + (size_t)page[i] * ((size_t)p.Hkv * VM_PAGE_TOKENS * p.D)
                                     + ((size_t)hk * VM_PAGE_TOKENS + pos[i] % VM_PAGE_TOKENS) * p.D;
                dst[da] = __float2bfloat16_rn(ya); dst[db] = __float2bfloat16_rn(yb);
            }
        }
    }
}

template <int NT, int PF, int WARPS, int TP, int EPI>
int launch(const SkinnyParams& p, int items, cudaStream_t stream) {
    vm_launch_pdl(skinny_direct_kernel<NT, PF, WARPS, TP, EPI>, dim3((items + TP - 1) / TP), dim3(WARPS * 32 + (p.squares ? 32 : 0)), 0, stream, p);
    return vm_launch_status();
}

// Blocks in flight: as many as leave two blocks of eight warps (one of 16) on an SM their registers.  More than four of a block of eight warps did not pay
// (6,144 x 2,048 at 8 rows: 5.9 us with four, 8.2 with six and one block fewer on the SM).
template <int NT, int EPI> int launch_rows(const SkinnyParams& p, int items, int warps, int tp, cudaStream_t stream) {
    const int per = (p.K / 32 + warps - 1) / warps;
    if constexpr (EPI == DIRECT_UNIT || EPI == DIRECT_STORE) {
        if (tp == 2) return per > 3 && NT == 1 ? launch<NT, (NT == 1 ? 4 : 3), 8, 2, EPI>(p, items, stream) : launch<NT, (NT == 4 ? 2 : 3), 8, 2, EPI>(p, items, stream);
    }
    if constexpr (NT < 4) {
        if (warps == 16) return per <= 3 ? launch<NT, 3, 16, 1, EPI>(p, items, stream) : launch<NT, (NT == 1 ? 6 : 4), 16, 1, EPI>(p, items, stream);
        if (per > 3) return launch<NT, 4, 8, 1, EPI>(p, items, stream);
    }
    return launch<NT, 3, 8, 1, EPI>(p, items, stream);
}

// Sixteen warps share K where the blocks do not cover the SMs and a warp of eight would take more than four blocks of K (576 x 1,536, 8 rows: 1.9 us
// against 2.2; 960 x 2,560: 2.7 / 3.7) or more than eight rows (960 x 960, 16 rows: 2.0 / 2.4).  Two pairs of column tiles a block where there are more
// pairs than SMs and K is at most 1,024 (2 x 1,536 x 576, 8 rows: 2.3 us against 2.8, the rows are fetched by half as many blocks); of longer rows a block
// would hold more weights than its registers (2 x 5,632 x 2,048: 11.2 / 9.2).
template <int EPI> int launch_direct(const SkinnyParams& p, int items, cudaStream_t stream) {
    const int sms = vm_sm_count();
    const int warps = items <= sms && (p.K > 1024 || p.M > 8) && p.M <= 16 ? 16 : 8;
    const int tp = (EPI == DIRECT_UNIT || EPI == DIRECT_STORE) && items > sms && p.K <= 1024 ? 2 : 1;
    if (p.M <= 8) return launch_rows<1, EPI>(p, items, warps, tp, stream);
    if (p.M <= 16) return launch_rows<2, EPI>(p, items, warps, tp, stream);
    return launch_rows<4, EPI>(p, items, warps, tp, stream);
}

}  // namespace

int vm_skinny_direct(const vmsk::SkinnyParams& p, int items, cudaStream_t stream) {
    if (p.M <= 0 || items <= 0) return 0;
    // (a residual product has no warp that joins squares, and no scale in its epilogue: its rows are plain)
    if (p.M > 32 || p.K <= 0 || p.K % 32 != 0 || (p.squares && (p.parts % 4 || p.epi == EPI_RESIDUAL))) return VM_ERR_UNSUPPORTED;
    switch (p.epi) {
        case EPI_STORE_BF16: case EPI_STORE_F32: return launch_direct<DIRECT_STORE>(p, items, stream);
        case EPI_RESIDUAL: return launch_direct<DIRECT_RESIDUAL>(p, items, stream);
        case EPI_SWIGLU: return launch_direct<DIRECT_UNIT>(p, items, stream);
        case EPI_ROPE_KV: return launch_direct<DIRECT_ROPE>(p, items, stream);
    }
    return VM_ERR_UNSUPPORTED;
}
