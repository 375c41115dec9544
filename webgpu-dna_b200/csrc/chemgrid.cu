// chemgrid.cu -- the reference's 'gpu' chemistry backend
// (src/shaders/chemistry.wgsl:1-334, driven by src/chemistry/schedule.ts:33-247
// and measure.ts): radicals diffuse in fixed time steps, a spatial hash of
// 1.5 nm cells finds neighbours, and pairs within the reaction radius react
// with a contact probability, each thread claiming both radicals with
// compare-and-swap (so, as in the reference, which of several competing
// pairs reacts depends on thread timing).  The 7-stage schedule (133 steps of
// diffuse / place / sort / react, plus the counts at each checkpoint) is
// captured once into a CUDA graph and replayed with one launch: the number of radicals
// and the key are read from memory (CgState), so calls of about the same size share it
// (a new batch of 20,000 radicals 5.7 -> 3.3 ms, of 530,000 15.1 -> 12.8; with each size and key
// captured anew, 2.2 ms of each call were the capture).  Without a graph the 133 steps'
// launches take 2 ms more than with one at every size.
//
// What bounds a step: 27 table lookups per radical, and at the common start of all
// tracks, where a reference cell holds hundreds of radicals, the pair tests.  The
// neighbours are therefore found in cells of half the reference's edge (0.75 nm,
// still above the largest reaction radius, so the same pairs are in contact and
// there are 6 times fewer to test), the radicals of a cell are stored side by side
// (a counting sort per step) instead of chained, and are read four at a time.
// Measured at 4096 x 1 keV (0.53 M radicals, all tracks from one point): 1680 us per step with
// lists of 1.5 nm cells, 160 us now.
//
// The reference's walk stops after 1024 entries of a 1.5 nm cell.  While no such cell
// (eight of 0.75 nm) holds more, no walk is stopped; the contacts found are rolled in the
// order of the lists (k_cg_react), so the results are theirs, up to which of several
// claims on one radical is the first.  A step with a fuller cell walks the lists as the
// reference does.
//
// Random numbers: Philox4x32-10 with counter (radical, step, 0, 6) and the
// call's key; the f32 Gaussians use this build's own log / sincos
// (dmath.cuh), so the CPU restatement reproduces every displacement.
#include "chemgrid.cuh"
#include "dmath.cuh"

namespace wg {

constexpr uint32_t CG_HASH = CG_HASH_SIZE;       // 2^23 buckets
constexpr float CG_CELL = 1.5f;                  // nm

__device__ __forceinline__ uint32_t cg_hash(int ix, int iy, int iz) {
    const uint32_t h = (uint32_t)(ix * 73856093) ^ (uint32_t)(iy * 19349663) ^ (uint32_t)(iz * 83492791);
    return h % CG_HASH;
}

__device__ __forceinline__ float cg_sigma_react(int a, int b) {
    if (a > b) { int t = a; a = b; b = t; }
    if (a == 0 && b == 0) return 0.44f;
    if (a == 0 && b == 1) return 0.57f;
    if (a == 0 && b == 2) return 0.45f;
    if (a == 1 && b == 1) return 0.54f;
    if (a == 1 && b == 2) return 0.61f;
    if (a == 1 && b == 3) return 0.47f;
    if (a == 2 && b == 2) return 0.34f;
    return 0.0f;
}

__device__ __forceinline__ float cg_pcontact(int a, int b) {
    if (a > b) { int t = a; a = b; b = t; }
    if (a == 0 && b == 0) return 0.376f;
    if (a == 0 && b == 1) return 0.980f;
    if (a == 0 && b == 2) return 0.511f;
    if (a == 1 && b == 1) return 0.125f;
    if (a == 1 && b == 2) return 0.455f;
    if (a == 1 && b == 3) return 0.538f;
    if (a == 2 && b == 2) return 0.216f;
    return 0.0f;
}

// product class: 1 = H2O2, 2 = H2, 3 = the e-aq + H3O+ -> H conversion
__device__ __forceinline__ int cg_product(int a, int b) {
    if (a > b) { int t = a; a = b; b = t; }
    if (a == 0 && b == 0) return 1;
    if (a == 1 && b == 1) return 2;
    if (a == 1 && b == 2) return 2;
    if (a == 1 && b == 3) return 3;
    if (a == 2 && b == 2) return 2;
    return 0;
}

// Box-Muller pair from two uniforms (gauss2, chemistry.wgsl:24-30)
__device__ __forceinline__ float2 cg_gauss2(float u1, float u2) {
    u1 = fmaxf(u1, 1e-10f);
    const float r = sqrtf(-2.0f * logf_pos(u1));
    float s, c;
    sincosf_(6.28318530f * u2, &s, &c);
    return make_float2(r * c, r * s);
}

// sample_init + init_thermal (chemistry.wgsl:92-101, 286-334)
__global__ void k_cg_init(const float4* rad, uint32_t n, uint32_t k0, uint32_t k1, float4* pos, uint32_t* alive,
                          CgState* st) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i == 0) { st->n = n; st->k0 = k0; st->k1 = k1; st->dense[0] = st->dense[1] = 0u; }
    if (i >= n) return;
    const float4 r = rad[i];
    int kind = (int)(__float2uint_rn(r.w) % 8u);
    float4 p = make_float4(r.x, r.y, r.z, (float)kind);
    alive[i] = 1u;
    const u4 w = philox(i, 0xffffffffu, 0u, 6u, k0, k1);
    float sigma = 0.0f;
    bool disp = true;
    if (kind == 0) sigma = 0.462f;
    else if (kind == 1) sigma = 1.764f;
    else if (kind == 2) sigma = 1.309f;
    else if (kind == 3) sigma = u01f(w.w) < 0.5f ? 0.462f : 0.0f;
    else if (kind == 5) { kind = 1; sigma = 0.0f; }
    else disp = false;
    if (disp) {
        const float2 g01 = cg_gauss2(u01f(w.x), u01f(w.y));
        const u4 w2 = philox(i, 0xfffffffeu, 0u, 6u, k0, k1);
        const float2 g23 = cg_gauss2(u01f(w2.x), u01f(w2.y));
        p.x = p.x + sigma * g01.x;
        p.y = p.y + sigma * g01.y;
        p.z = p.z + sigma * g23.x;
        p.w = (float)kind;
    }
    pos[i] = p;
}

constexpr float CG_FINE = 0.75f;                 // nm
constexpr uint32_t CG_NONE = 0xffffffffu;
constexpr uint32_t CG_WALK = 1024;               // the reference's bound on a walk through a cell
__device__ __forceinline__ int cg_fine(float x) { return (int)floorf(x / CG_FINE); }

__device__ __forceinline__ int cg_cell(float x) { return (int)floorf(x / CG_CELL); }
__device__ __forceinline__ uint32_t cg_list(float4 p) { return cg_hash(cg_cell(p.x), cg_cell(p.y), cg_cell(p.z)); }

// 1) diffuse (chemistry.wgsl:32-56) and take a place in the fine cell's bucket.  After a
//    step with lists, each radical empties the one it was in (it has not moved since).
__global__ void k_cg_diffuse(float4* pos, const uint32_t* alive, float dt, uint32_t step, uint32_t* tab, uint32_t* cell,
                             uint32_t* rank, CgState* st, int* head) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i == 0) { st->placed = 0u; st->dense[step & 1u] = 0u; }
    if (i >= st->n) return;
    if (st->dense[(step + 1) & 1u]) head[cg_list(pos[i])] = -1;
    if (alive[i] == 0u) { cell[i] = CG_NONE; return; }
    float4 p = pos[i];
    const int kind = (int)rintf(p.w);
    float D = 0.0f;
    if (kind == 0) D = 2.2f;
    else if (kind == 1) D = 4.9f;
    else if (kind == 2) D = 7.0f;
    else if (kind == 3) D = 9.0f;
    if (kind >= 0 && kind <= 3) {
        const float sigma = sqrtf(2.0f * D * dt);
        const u4 w = philox(i, step, 0u, 6u, st->k0, st->k1);
        const float2 g01 = cg_gauss2(u01f(w.x), u01f(w.y));
        const float2 g23 = cg_gauss2(u01f(w.z), u01f(w.w));
        p.x += sigma * g01.x;
        p.y += sigma * g01.y;
        p.z += sigma * g23.x;
        pos[i] = p;
    }
    const uint32_t h = cg_hash(cg_fine(p.x), cg_fine(p.y), cg_fine(p.z));
    cell[i] = h;
    rank[i] = atomicAdd(&tab[h], 1u);
}

// count of a bucket whose word may already hold its first entry as well
__device__ __forceinline__ uint32_t cg_count(uint32_t v) { return (v >> 23) ? v >> 23 : v; }

// 2) the first radical of each bucket reserves the bucket's entries: one atomic
//    per block, so buckets keep the order of the tracks.  The table word becomes
//    first entry | count << 23.  A fine cell with more than an eighth of CG_WALK has
//    its coarse cell counted.
constexpr int CG_RB = 512;
__global__ void __launch_bounds__(CG_RB) k_cg_reserve(const float4* pos, uint32_t* tab, const uint32_t* cell,
                                                      const uint32_t* rank, CgState* st, uint32_t step) {
    __shared__ uint32_t wsum[CG_RB / 32], s_base;
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    const int lane = threadIdx.x & 31, wl = threadIdx.x >> 5;
    const uint32_t h = i < st->n ? cell[i] : CG_NONE;
    const bool lead = h != CG_NONE && rank[i] == 0u;
    const uint32_t c = lead ? tab[h] : 0u;
    uint32_t off = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) { const uint32_t v = __shfl_up_sync(0xffffffffu, off, o); if (lane >= o) off += v; }
    if (lane == 31) wsum[wl] = off;
    __syncthreads();
    if (wl == 0) {
        const uint32_t own = lane < CG_RB / 32 ? wsum[lane] : 0u;
        uint32_t v = own;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) { const uint32_t u = __shfl_up_sync(0xffffffffu, v, o); if (lane >= o) v += u; }
        if (lane < CG_RB / 32) wsum[lane] = v - own;
        if (lane == 31) s_base = v ? atomicAdd(&st->placed, v) : 0u;
    }
    __syncthreads();
    if (!lead) return;
    bool dense = c > 511u;                           // does not fit the word
    if (c > CG_WALK / 8 && !dense) {
        const float4 p = pos[i];
        const int ix = cg_fine(p.x) & ~1, iy = cg_fine(p.y) & ~1, iz = cg_fine(p.z) & ~1;
        uint32_t sum = 0;
        for (int o = 0; o < 8; ++o)
            sum += cg_count(*(volatile uint32_t*)&tab[cg_hash(ix + (o & 1), iy + ((o >> 1) & 1), iz + (o >> 2))]);
        dense = sum > CG_WALK;
    }
    if (dense) st->dense[step & 1u] = 1u;
    tab[h] = (s_base + wsum[wl] + off - c) | (min(c, 511u) << 23);
}

// 3) radicals in bucket order; the other table is emptied for the next step.  A step with
//    an overfull cell also builds the reference's lists (build_hash, chemistry.wgsl:111-122).
//    Clearing the heads and building the lists in launches of their own cost every ordinary
//    step two that return at once, and building them in k_cg_react slowed that kernel (530,000
//    radicals, a call: 12.4 ms with the launches, 14.2 with k_cg_react, 12.3 so).  Such a step
//    has no use for the bucket order: with 1200 radicals that stay in one cell a call of
//    5 million takes 466 ms (488 with the order made all the same, and with 592 blocks walking
//    the lists; 480 by lists alone).
__global__ void k_cg_sort(const float4* pos, const uint32_t* tab, const uint32_t* cell, const uint32_t* rank, float4* sorted,
                          uint32_t* tab_old, const uint32_t* cell_old, const CgState* st, uint32_t step, int* head, int* next) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= st->n) return;
    if (cell_old) { const uint32_t o = cell_old[i]; if (o != CG_NONE) tab_old[o] = 0u; }
    const uint32_t h = cell[i];
    if (h == CG_NONE) return;                        // dead: no list leads to it
    const float4 p = pos[i];
    if (st->dense[step & 1u]) { next[i] = atomicExch(&head[cg_list(p)], (int)i); return; }
    const uint32_t kind = (uint32_t)(int)rintf(p.w) & 7u;
    sorted[(tab[h] & 0x7fffffu) + rank[i]] = make_float4(p.x, p.y, p.z, __uint_as_float(i | (kind << 23)));
}

// a pair within R_max: the contact test (with i's kind when its walk began and j's kind
// of now, as the reference reads them), the roll, the claim.  0: go on, 1: radical i is
// done with this step
__device__ __forceinline__ int cg_contact(float4* pos, uint32_t* alive, uint32_t i, int ki, uint32_t j, float d2, uint32_t step,
                                          const CgState* st, uint32_t& draw, u4& w, uint32_t* prod) {
    if (alive[j] == 0u) return 0;
    const int kj = (int)rintf(pos[j].w);
    if (kj < 0 || kj > 3) return 0;
    const float R = cg_sigma_react(ki, kj);
    if (R <= 0.0f || d2 > R * R) return 0;
    if ((draw & 3u) == 0u) w = philox(i, step, 1u + (draw >> 2), 6u, st->k0, st->k1);
    const uint32_t word = (draw & 3u) == 0u ? w.x : (draw & 3u) == 1u ? w.y : (draw & 3u) == 2u ? w.z : w.w;
    draw++;
    if (u01f(word) >= cg_pcontact(ki, kj)) return 0;
    if (atomicCAS(&alive[i], 1u, 0u) != 1u) return 1;
    if (atomicCAS(&alive[j], 1u, 0u) != 1u) { atomicExch(&alive[i], 1u); return 0; }
    const int pr = cg_product(ki, kj);
    if (pr == 1) atomicAdd(&prod[0], 1u);
    else if (pr == 2) atomicAdd(&prod[1], 1u);
    else if (pr == 3) {
        const uint32_t e = ki == 1 ? i : j;         // the e-aq becomes an H
        pos[e].w = 2.0f;
        atomicExch(&alive[e], 1u);
    }
    return 1;
}

// 4) react (chemistry.wgsl:194-266): contact within the reaction radius, a
//    contact-probability roll from the radical's step stream, claim both
//    radicals with compare-and-swap.  The pair belongs to its lower index.  Threads
//    take the radicals in index order: which of several contacts is claimed
//    depends on when threads run, and cell order shifts the yields of a crowded
//    origin by 0.1 % for 5 % of the time.
//    The first contact that passes its roll wins, so the order of the rolls decides which
//    kind of pair reacts.  It is the lists': the 27 cells of 1.5 nm one after another, a
//    cell's radicals by falling index.  The contacts found in the 0.75 nm cells are therefore
//    kept by their place in that walk (CG_KEEP at a time; a radical whose rolls all fail
//    looks through the cells again for the ones after) before the first roll.  A cell that
//    shares its bucket with another of the walk is met at both places, as in the lists:
//    (-1, -1, z) and (1, 1, z) always do.  (Not the lists': a position that is not a number is
//    in contact with nothing here.)
//    Yields after 1 us against claims in radical order, H2O2 and H2, mean of 32 inputs of
//    30,000 radicals in 15 clusters of sigma 0.4 nm (40 of 0.5 nm): lists -2.7 and -1.9 %
//    (-1.6 and -0.8), rolls in the order of the 0.75 nm cells -4.2 and -2.9 (-3.2 and -2.2),
//    now +1.0 and +0.4 (+1.6 and +0.7).  CG_KEEP 4 and 8, a call of 530,000 radicals: 12.7 ms
//    both; 40 clusters 2.2 and 1.6 % of H2O2; in the cells' order 11.6 ms.
//    The kept contacts cost 13 registers, and so one of 5 blocks per SM: 700 x 5 keV 12.5 ms in the
//    cells' order, 13.8 now (lists 20.6).  In shared memory at 48 registers 13.4, but the 15
//    clusters 32 ms instead of 18.5; a first look for any contact at all 14.3.
constexpr uint32_t CG_LAST = 0x7fffffu;          // a contact's key: place << 23 | CG_LAST - index
constexpr int CG_KEEP = 8;

__global__ void k_cg_react(float4* pos, uint32_t* alive, const uint32_t* tab, const float4* sorted, const CgState* st,
                           uint32_t step, uint32_t* prod) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= st->n || st->dense[step & 1u] || alive[i] == 0u) return;
    const float4 me = pos[i];
    const int ki = (int)rintf(me.w);
    if (ki < 0 || ki > 3) return;
    const int ix = cg_fine(me.x), iy = cg_fine(me.y), iz = cg_fine(me.z);
    const int cx = cg_cell(me.x), cy = cg_cell(me.y), cz = cg_cell(me.z);
    // largest squared distance of a contact by the other's kind when it was sorted (an e-aq may
    // have become an H since)
    float r2k[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const float r = k == 1 ? fmaxf(cg_sigma_react(ki, 1), cg_sigma_react(ki, 2)) : cg_sigma_react(ki, k);
        r2k[k] = r > 0.0f ? r * r : -1.0f;
    }
    const float r2m = fmaxf(fmaxf(r2k[0], r2k[1]), fmaxf(r2k[2], r2k[3]));
    uint32_t draw = 0, from = 0;
    u4 w = {0, 0, 0, 0};
    for (;;) {
        // the first CG_KEEP contacts from `from` on: place of the cell in the walk, falling index
        uint32_t key[CG_KEEP];
#pragma unroll
        for (int k = 0; k < CG_KEEP; ++k) key[k] = CG_NONE;
        for (int dz = -1; dz <= 1; ++dz)
            for (int dy = -1; dy <= 1; ++dy) {
                uint32_t word[3];                                // three lookups in flight
#pragma unroll
                for (int dx = 0; dx < 3; ++dx) word[dx] = tab[cg_hash(ix + dx - 1, iy + dy, iz + dz)];
#pragma unroll 1
                for (int dx = 0; dx < 3; ++dx) {
                    const uint32_t v = dx == 0 ? word[0] : dx == 1 ? word[1] : word[2];
                    const float4* S = sorted + (v & 0x7fffffu);
                    // four entries in flight
                    for (int c = (int)(v >> 23) - 1; c >= 0; c -= 4) {
                        float d2[4];
                        uint32_t jw[4];
#pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            const float4 q = S[max(c - u, 0)];
                            const float ddx = me.x - q.x, ddy = me.y - q.y, ddz = me.z - q.z;
                            d2[u] = c >= u ? ddx * ddx + ddy * ddy + ddz * ddz : 1e30f;
                            jw[u] = __float_as_uint(q.w);
                        }
                        if (fminf(fminf(d2[0], d2[1]), fminf(d2[2], d2[3])) > r2m) continue;
                        uint32_t m = 0;
#pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            const uint32_t kj = jw[u] >> 23;
                            const float lim = kj == 0u ? r2k[0] : kj == 1u ? r2k[1] : kj == 2u ? r2k[2] : kj == 3u ? r2k[3] : -1.0f;
                            if (d2[u] <= lim && (jw[u] & CG_LAST) > i) m |= 1u << u;
                        }
#pragma unroll 1
                        for (; m; m &= m - 1u) {
                            const float4 q = S[c - (__ffs(m) - 1)];
                            const uint32_t low = CG_LAST - (__float_as_uint(q.w) & CG_LAST);
                            const uint32_t hq = cg_list(q);
                            uint32_t place = 0;
#pragma unroll 1
                            for (int z = -1; z <= 1; ++z)
#pragma unroll 1
                                for (int y = -1; y <= 1; ++y)
#pragma unroll 1
                                    for (int x = -1; x <= 1; ++x, ++place) {
                                        if (cg_hash(cx + x, cy + y, cz + z) != hq) continue;
                                        uint32_t add = place << 23 | low;
                                        bool have = add < from;
#pragma unroll
                                        for (int k = 0; k < CG_KEEP; ++k) have |= add == key[k];
                                        if (have) continue;      // (two 0.75 nm cells of one bucket find it twice)
#pragma unroll
                                        for (int k = 0; k < CG_KEEP; ++k) {
                                            const uint32_t old = key[k];
                                            key[k] = min(old, add);
                                            add = max(old, add);
                                        }
                                    }
                        }
                    }
                }
            }
#pragma unroll 1
        for (int k = 0; k < CG_KEEP; ++k) {
            const uint32_t first = key[0], j = CG_LAST - (first & CG_LAST);
            if (first == CG_NONE) return;
#pragma unroll
            for (int q = 1; q < CG_KEEP; ++q) key[q - 1] = key[q];
            from = first + 1u;
            const float4 q = pos[j];
            const float ddx = me.x - q.x, ddy = me.y - q.y, ddz = me.z - q.z;
            if (cg_contact(pos, alive, i, ki, j, ddx * ddx + ddy * ddy + ddz * ddz, step, st, draw, w, prod)) return;
        }
    }
}

// Steps with an overfull cell: the reference's walk (chemistry.wgsl:194-266), at most
// 1024 entries of a list deep.
__global__ void k_cg_react_list(const CgState* st, float4* pos, uint32_t* alive, const int* head, const int* next,
                                uint32_t step, uint32_t* prod) {
    if (!st->dense[step & 1u]) return;
    const uint32_t n = st->n;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        if (alive[i] == 0u) continue;
        const float4 pi = pos[i];
        const int ki = (int)rintf(pi.w);
        if (ki < 0 || ki > 3) continue;
        const int ix = cg_cell(pi.x), iy = cg_cell(pi.y), iz = cg_cell(pi.z);
        uint32_t draw = 0;
        u4 w = {0, 0, 0, 0};
        bool done = false;
        for (int c = 0; c < 27 && !done; ++c) {
            int j = head[cg_hash(ix + c % 3 - 1, iy + c / 3 % 3 - 1, iz + c / 9 - 1)];
            for (uint32_t it = 0; it < 1024u && j >= 0 && !done; ++it) {
                const uint32_t ju = (uint32_t)j;
                j = next[ju];
                if (ju <= i) continue;
                const float4 pj = pos[ju];
                const float ddx = pi.x - pj.x, ddy = pi.y - pj.y, ddz = pi.z - pj.z;
                done = cg_contact(pos, alive, i, ki, ju, ddx * ddx + ddy * ddy + ddz * ddz, step, st, draw, w, prod) != 0;
            }
        }
    }
}

// count_alive (chemistry.wgsl:270-281) into checkpoint slot k: OH, e-aq, H
// alive, then the running H2O2 and H2 product counts
__global__ void k_cg_count(const float4* pos, const uint32_t* alive, const CgState* st, const uint32_t* prod,
                           uint32_t* out) {
    __shared__ uint32_t s[3];
    const uint32_t n = st->n;
    if (threadIdx.x < 3) s[threadIdx.x] = 0;
    __syncthreads();
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        if (alive[i] == 0u) continue;
        const int kind = (int)rintf(pos[i].w);
        if (kind >= 0 && kind <= 2) atomicAdd(&s[kind], 1u);
    }
    __syncthreads();
    if (threadIdx.x < 3 && s[threadIdx.x]) atomicAdd(&out[threadIdx.x], s[threadIdx.x]);
    if (blockIdx.x == 0 && threadIdx.x == 0) { out[3] = prod[0]; out[4] = prod[1]; }
}

// The schedule of schedule.ts:38-46: [dt ns, steps]
static const float CG_DT[7] = {0.0001f, 0.001f, 0.005f, 0.05f, 0.5f, 3.0f, 30.0f};
static const int CG_NS[7] = {10, 9, 18, 18, 18, 30, 30};

// Blocks of 256 for n radicals, rounded up to one of eight sizes per factor of two, so that
// batches of about the same size (a spectrum's next seed) find their schedule captured.
uint32_t cg_blocks(uint32_t n) {
    const uint32_t nb = (n + 255) / 256;
    uint32_t unit = 1;
    while (unit * 16 <= nb) unit *= 2;
    return (nb + unit - 1) / unit * unit;
}

cudaError_t cg_run(const CgArgs& a, cudaStream_t s, cudaGraphExec_t* cache, CgGraphKey* key) {
    const uint32_t n = a.n;
    const unsigned nb = cg_blocks(n);
    cudaError_t e;
    k_cg_init<<<nb, 256, 0, s>>>(a.rad, n, a.k0, a.k1, a.pos, a.alive, a.st);
    { cudaError_t me_ = cudaMemsetAsync(a.counts, 0, 8 * 5 * sizeof(uint32_t), s); if (me_ != cudaSuccess) return me_; }
    { cudaError_t me_ = cudaMemsetAsync(a.prod, 0, 2 * sizeof(uint32_t), s); if (me_ != cudaSuccess) return me_; }
    k_cg_count<<<296, 256, 0, s>>>(a.pos, a.alive, a.st, a.prod, a.counts);
    if ((e = cudaMemsetAsync(a.tab, 0, 2 * (size_t)CG_HASH * sizeof(uint32_t), s)) != cudaSuccess) return e;
    if ((e = cudaMemsetAsync(a.head, 0xff, (size_t)CG_HASH * sizeof(int), s)) != cudaSuccess) return e;
    // the schedule as one graph; rebuilt when the buffers or the grid sizes change
    CgGraphKey want;
    memset(&want, 0, sizeof want);
    want.pos = a.pos; want.sorted = a.sorted; want.alive = a.alive; want.tab = a.tab; want.cell = a.cell;
    want.rank = a.rank; want.prod = a.prod; want.counts = a.counts; want.head = a.head; want.next = a.next;
    want.st = a.st; want.nb = nb; want.cap = a.cap;
    if (!*cache || memcmp(key, &want, sizeof want) != 0) {
        if (*cache) { cudaGraphExecDestroy(*cache); *cache = nullptr; }
        cudaStream_t cs;
        if ((e = cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking)) != cudaSuccess) return e;
        cudaGraph_t g;
        if ((e = cudaStreamBeginCapture(cs, cudaStreamCaptureModeThreadLocal)) != cudaSuccess) { cudaStreamDestroy(cs); return e; }
        uint32_t step = 0;
        for (int stage = 0; stage < 7; ++stage) {
            for (int k = 0; k < CG_NS[stage]; ++k) {
                ++step;
                uint32_t *tab = a.tab + (size_t)(step & 1u) * CG_HASH, *tab_old = a.tab + (size_t)((step + 1) & 1u) * CG_HASH;
                uint32_t *cell = a.cell + (size_t)(step & 1u) * a.cap, *cell_old = a.cell + (size_t)((step + 1) & 1u) * a.cap;
                k_cg_diffuse<<<nb, 256, 0, cs>>>(a.pos, a.alive, CG_DT[stage], step, tab, cell, a.rank, a.st, a.head);
                k_cg_reserve<<<(nb * 256 + CG_RB - 1) / CG_RB, CG_RB, 0, cs>>>(a.pos, tab, cell, a.rank, a.st, step);
                k_cg_sort<<<nb, 256, 0, cs>>>(a.pos, tab, cell, a.rank, a.sorted, tab_old, step > 1 ? cell_old : nullptr,
                                              a.st, step, a.head, a.next);
                k_cg_react<<<nb, 256, 0, cs>>>(a.pos, a.alive, tab, a.sorted, a.st, step, a.prod);
                k_cg_react_list<<<nb < 1184 ? nb : 1184, 256, 0, cs>>>(a.st, a.pos, a.alive, a.head, a.next, step, a.prod);
            }
            k_cg_count<<<296, 256, 0, cs>>>(a.pos, a.alive, a.st, a.prod, a.counts + 5 * (stage + 1));
        }
        e = cudaStreamEndCapture(cs, &g);
        cudaStreamDestroy(cs);
        if (e != cudaSuccess) return e;
        e = cudaGraphInstantiate(cache, g, 0);
        cudaGraphDestroy(g);
        if (e != cudaSuccess) { *cache = nullptr; return e; }
        *key = want;
    }
    e = cudaGraphLaunch(*cache, s);
    if (e != cudaSuccess) return e;
    return cudaGetLastError();
}

}  // namespace wg
