// chemgrid.cuh -- the grid-hash diffusion-reaction chemistry backend.
#pragma once
#include <cstdint>
#include <cstring>
#include <cuda_runtime.h>

namespace wg {

struct CgState {
    uint32_t placed;         // entries in the cell-ordered copy
    uint32_t dense[2];       // even and odd steps: a cell too full for it
    uint32_t n, k0, k1;      // the call's radicals and key
};

struct CgArgs {
    const float4* rad;       // the first n rad_buf entries
    uint32_t n, k0, k1;
    uint32_t cap;            // the arrays' size, at least n
    float4* pos;             // n: x, y, z, kind
    uint32_t* alive;         // n
    uint32_t* tab;           // 2 x 2^23 buckets, for odd and even steps: entries, then first entry and count
    uint32_t* cell;          // 2 x cap: bucket of each radical in the step's grid
    uint32_t* rank;          // n: its place in the bucket
    float4* sorted;          // n: x, y, z, index and kind in bucket order
    int* head;               // 2^23 list heads and
    int* next;               // n links, for steps with an overfull cell
    uint32_t* prod;          // 2: H2O2, H2 made
    uint32_t* counts;        // 8 x 5: t = 0 and the 7 checkpoints
    CgState* st;
};

// what the captured schedule depends on (compared as bytes: no padding)
struct CgGraphKey {
    float4 *pos, *sorted;
    uint32_t *alive, *tab, *cell, *rank, *prod, *counts;
    int *head, *next;
    CgState* st;
    uint32_t nb, cap;
};

constexpr uint32_t CG_HASH_SIZE = 8388608u;
constexpr uint32_t CG_CHEM_N = 8000000u;   // CHEM_N, src/physics/constants.ts:57

uint32_t cg_blocks(uint32_t n);
cudaError_t cg_run(const CgArgs& a, cudaStream_t s, cudaGraphExec_t* cache, CgGraphKey* key);

}  // namespace wg
