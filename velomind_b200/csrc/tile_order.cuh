// Which tile of query rows and which head a CTA of a prompt's attention takes.
//
// The tiles of a causal prompt see one key block, two, three ...: dealt out in their order along the prompt, one SM gets long tiles only and another short ones
// (2,048 tokens, 9 heads in tiles of 64 rows: 288 CTAs, all resident, 12 to 52 key blocks an SM, 33 on average).  So the host lists a step's tiles by their number
// of blocks, the longest first (shape only: new tokens per sequence), and the CTAs, which the GPU deals out to its SMs in turn, take them forwards and
// backwards from wave to wave.  The list rides along as a kernel argument, two bytes a tile, so that no CTA walks over the sequences' offsets (a chain of loads)
// either.  Steps of more tiles than it holds keep that walk and take a prompt's last tiles first: they are many waves long.  A step of one tile gains nothing and pays
// 0.1 to 0.3 us (a prompt of 33 to 64 tokens, 9 heads of 64 3.6 -> 3.9; without the list 3.8, so most of it is the kernel's other code).
#pragma once
#include "common.cuh"

constexpr int VM_TILES_LISTED = 256;

struct VmTiles {
    int n, sms;                                          // n = 0: not listed
    unsigned short where[VM_TILES_LISTED];               // sequence << 8 | tile of the sequence
};

// host_cu_tokens [B + 1] on the host, or null: no list
static inline VmTiles vm_list_tiles(const int* host_cu_tokens, int B, int rows, int n_tiles) {
    VmTiles t;
    t.n = 0;
    t.sms = vm_sm_count();
    if (host_cu_tokens == nullptr || n_tiles > VM_TILES_LISTED || t.sms <= 0 || B > 256) return t;
    int place[VM_TILES_LISTED + 1] = {}, total = 0;      // tiles of each length, then where the next of that length goes
    for (int b = 0; b < B; ++b) {
        const int k = (host_cu_tokens[b + 1] - host_cu_tokens[b] + rows - 1) / rows;
        if (k < 0 || total + k > n_tiles) return t;
        for (int i = 0; i < k; ++i) ++place[i];
        total += k;
    }
    if (total != n_tiles) return t;
    for (int i = VM_TILES_LISTED, before = 0; i >= 0; --i) { const int here = place[i]; place[i] = before; before += here; }
    for (int b = 0; b < B; ++b)
        for (int i = 0; host_cu_tokens[b] + i * rows < host_cu_tokens[b + 1]; ++i) t.where[place[i]++] = (unsigned short)(b << 8 | i);
    t.n = n_tiles;
    return t;
}

// The tile and the head of this CTA of a grid (tiles, heads); false: none.  cu_tokens [B + 1] on the device.
__device__ __forceinline__ bool vm_tile_of(const VmTiles& tiles, const int* __restrict__ cu_tokens, int B, int rows, int& seq, int& t0, int& n_rows, int& head) {
    if (tiles.n > 0) {
        const int items = gridDim.x * gridDim.y, turn = blockIdx.y * gridDim.x + blockIdx.x, wave = turn / tiles.sms, first = wave * tiles.sms;
        const int item = wave & 1 ? first + min(tiles.sms, items - first) - 1 - (turn - first) : turn;
        const int k = item / gridDim.y;
        head = item - k * gridDim.y;
        seq = tiles.where[k] >> 8;
        t0 = cu_tokens[seq] + (tiles.where[k] & 255) * rows;
        n_rows = min(rows, cu_tokens[seq + 1] - t0);
        return true;
    }
    int tile = gridDim.x - 1 - blockIdx.x;               // (the last tiles of a sequence see the most keys: they are started first)
    head = blockIdx.y;
    for (seq = 0; seq < B; ++seq) {
        const int a = cu_tokens[seq], b = cu_tokens[seq + 1], nt = (b - a + rows - 1) / rows;
        if (tile < nt) { t0 = a + tile * rows; n_rows = min(rows, b - t0); return true; }
        tile -= nt;
    }
    return false;
}
