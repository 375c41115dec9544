// scoring.cu -- SSB / DSB scoring on the B-DNA fibre grid.
//
// Results are bit-identical to src/scoring/ssb-dsb.ts of allaunthefox/webgpu-dna
// (scoreDirectSSB_events :135-217, scoreIndirectSSB :43-121, clusterDSB
// :348-407, makeSsbRng :421-427) evaluated with JavaScript number semantics.
// The reference is a sequential loop; here every entry is scored in parallel:
//
//  1. k_find: a warp per segment of 512 entries, in order.  The reference's
//     skip-by-2 walk visits entry i iff its distance from the start of its run of
//     equal positions is even, that is iff i has the parity of that start.  The
//     entries within reach of a backbone (a few in ten thousand) are listed in
//     order; those before the segment's first run start wait for the parity
//     that comes in.
//  2. k_draw: every block sums the draws of the segments before its own, each
//     thread then walks one segment's list: the LCG state after k steps is an affine
//     map (1664525 s + 1013904223 mod 2^32) raised to k by squaring, and one step
//     per draw from there on; a draw below p sets the hit byte (atomicOr, counted
//     once).
//
// What bounds it: the 16 bytes per entry that k_find reads.  An f32 test of the
// distance to the nearest fibre axis keeps all but the listed entries out of the
// f64 geometry, and nothing is written per entry.
// Measured on 5.3 M entries of 4096 x 10 keV: 203 us with an info word per entry and
// block-wide scans over 1024-entry tiles (k_prep 33, k_tiles 74, k_tilescan 22,
// k_apply 70, launches), 45 us now (k_find 29, k_draw 16).
//
// clusterDSB: one block per fibre collects the strand-0 / strand-1 hit lists
// in order and pairs them greedily; the expected-DSB sum uses the host's pow.
#include "scoring.cuh"

namespace wg {


constexpr int SEG = (int)SCORE_SEG;

__device__ __forceinline__ double js_round(double x) {
    double f = floor(x);
    return (x - f >= 0.5) ? f + 1.0 : f;
}

// nearest backbone within r_d (ssb-dsb.ts:73-106); returns hit index or -1
__device__ __forceinline__ long long near_backbone(const DnaDev& d, double x, double y, double z,
                                                   double r_d, int* cand) {
    double x_half = ((double)d.n_bp_per - 1) * d.rise * 0.5;
    double rise_inv = 1 / d.rise;
    double grid_off = -(((double)d.grid_N - 1) * d.spacing) * 0.5;
    double inv_sp = 1 / d.spacing;
    *cand = 0;
    if (x < -x_half - r_d || x > x_half + r_d) return -1;
    double fi = js_round((y - grid_off) * inv_sp);
    double fj = js_round((z - grid_off) * inv_sp);
    if (fi < 0 || fi >= d.grid_N || fj < 0 || fj >= d.grid_N) return -1;
    uint32_t fiber = (uint32_t)fi * d.grid_N + (uint32_t)fj;
    double y_rel = y - (double)d.fy[fiber];
    double z_rel = z - (double)d.fz[fiber];
    double r2 = y_rel * y_rel + z_rel * z_rel;
    double outer = d.r_bb + r_d;
    if (r2 > outer * outer) return -1;
    *cand = 1;
    double bp_est = js_round((x + x_half) * rise_inv);
    double b0 = bp_est - 2 > 0 ? bp_est - 2 : 0;
    double b1 = bp_est + 2 < (double)d.n_bp_per - 1 ? bp_est + 2 : (double)d.n_bp_per - 1;
    double best = __longlong_as_double(0x7ff0000000000000ll);
    long long best_bp = -1;
    int best_s = -1;
    for (double bb = b0; bb <= b1; bb += 1) {
        long long b = (long long)bb;
        double dx = x - (d.x0 + bb * d.rise);
        double dy0 = y_rel - (double)d.rbb0[2 * b], dz0 = z_rel - (double)d.rbb0[2 * b + 1];
        double d20 = dx * dx + dy0 * dy0 + dz0 * dz0;
        if (d20 < best) { best = d20; best_bp = b; best_s = 0; }
        double dy1 = y_rel - (double)d.rbb1[2 * b], dz1 = z_rel - (double)d.rbb1[2 * b + 1];
        double d21 = dx * dx + dy1 * dy1 + dz1 * dz1;
        if (d21 < best) { best = d21; best_bp = b; best_s = 1; }
    }
    if (!(best < r_d * r_d)) return -1;
    return (long long)fiber * d.n_bp_per + best_bp + (long long)best_s * d.n_bp;
}

// False only if the entry is certainly beyond reach of every fibre axis: the f32 offset
// from the nearest axis has an error of at most (|grid_off| + 3 |y - grid_off| + sp / 2) 2^-24,
// below 0.05 nm for |y|, |z| and |grid_off| up to 100 um, and `far` adds that to the reach (it
// is infinite on a wider grid).  A NaN goes on to the f64 geometry.
__device__ __forceinline__ bool maybe_near(float y, float z, float grid_off, float inv_sp, float sp, float far) {
    const float u = (y - grid_off) * inv_sp, v = (z - grid_off) * inv_sp;
    const float dy = fabsf(u - rintf(u)) * sp, dz = fabsf(v - rintf(v)) * sp;
    return (dy <= far && dz <= far) || !(dy + dz >= 0.0f) || fmaxf(fabsf(y), fabsf(z)) > 1e5f;
}

// A segment's summary: listed draws (resolved, waiting with even and odd index) and
// candidates (near a fibre axis, ssb-dsb.ts:183) the same way, ten bits each, then
// whether a run starts in the segment and the parity of its last run start.
// List words: bit31 waiting, bit30 parity of the index, bits 0..28 hit index.
__device__ __forceinline__ uint32_t fld(unsigned long long v, int k) { return (uint32_t)(v >> (10 * k)) & 1023u; }

constexpr int FB = 256;
__global__ void __launch_bounds__(FB) k_find(const float4* rad, const uint32_t* alive, unsigned long long n, DnaDev d,
                                             double r_d, int dedupe, uint32_t* list, unsigned long long* seg,
                                             unsigned long long* cnt) {
    const int lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1u;
    if (blockIdx.x == 0 && threadIdx.x < 8) cnt[threadIdx.x] = 0ull;
    const unsigned long long q = (unsigned long long)blockIdx.x * (FB / 32) + (threadIdx.x >> 5);
    const unsigned long long a = q * SEG;
    if (a >= n) return;
    const float grid_off = (float)(-(((double)d.grid_N - 1) * d.spacing) * 0.5), sp = (float)d.spacing;
    const float inv_sp = (float)(1 / d.spacing);
    const float far = grid_off >= -1e5f ? (float)(d.r_bb + r_d) + 0.05f : __int_as_float(0x7f800000);
    uint32_t f[6] = {0, 0, 0, 0, 0, 0}, len = 0;
    bool open = true;                             // no run has started in the segment yet
    uint32_t par = 0;                             // parity of the last run start
    float4 last = make_float4(0.f, 0.f, 0.f, 0.f);
    if (dedupe && a > 0) last = rad[a - 1];
    constexpr int U = 4;
    for (int c = 0; c < SEG; c += 32 * U) {
        if (a + c >= n) break;
        float4 e[U];
        uint32_t al[U];
#pragma unroll
        for (int k = 0; k < U; ++k) {
            const unsigned long long i = a + c + 32 * k + lane;
            e[k] = i < n ? __ldcs(rad + i) : make_float4(0.f, 0.f, 0.f, 0.f);
            al[k] = alive ? (i < n ? alive[i] : 0u) : 1u;
        }
#pragma unroll
        for (int k = 0; k < U; ++k) {
            const unsigned long long i = a + c + 32 * k + lane;
            const bool in = i < n;
            unsigned brk = 0xffffffffu;
            if (dedupe) {
                float4 p;
                p.x = __shfl_up_sync(0xffffffffu, e[k].x, 1); p.y = __shfl_up_sync(0xffffffffu, e[k].y, 1);
                p.z = __shfl_up_sync(0xffffffffu, e[k].z, 1);
                if (lane == 0) p = last;
                brk = __ballot_sync(0xffffffffu, in && (i == 0 || !(p.x == e[k].x && p.y == e[k].y && p.z == e[k].z)));
                last.x = __shfl_sync(0xffffffffu, e[k].x, 31); last.y = __shfl_sync(0xffffffffu, e[k].y, 31);
                last.z = __shfl_sync(0xffffffffu, e[k].z, 31);
            }
            const bool look = in && al[k] != 0u && (!alive || js_round((double)e[k].w) == 0.0) &&      // OH only
                              maybe_near(e[k].y, e[k].z, grid_off, inv_sp, sp, far);
            if (__any_sync(0xffffffffu, look)) {
                int cand = 0;
                long long h = -1;
                if (look) h = near_backbone(d, e[k].x, e[k].y, e[k].z, r_d, &cand);
                const unsigned b = brk & (lt | (1u << lane));      // run starts up to this entry
                const uint32_t odd = (uint32_t)lane & 1u;          // a, c and 32 k are even
                const bool wait = open && b == 0u;
                const uint32_t start = b ? (uint32_t)(31 - __clz(b)) & 1u : par;
                const bool seen = cand && (wait || start == odd);
                const bool draw = seen && h >= 0;
                const unsigned m = __ballot_sync(0xffffffffu, draw);
                if (draw)
                    list[a + len + __popc(m & lt)] = (wait ? 0x80000000u | (odd << 30) : 0u) | (uint32_t)h;
                len += __popc(m);
                const unsigned w = __ballot_sync(0xffffffffu, wait), s = __ballot_sync(0xffffffffu, seen);
                f[0] += __popc(m & ~w); f[1] += __popc(m & w & 0x55555555u); f[2] += __popc(m & w & 0xaaaaaaaau);
                f[3] += __popc(s & ~w); f[4] += __popc(s & w & 0x55555555u); f[5] += __popc(s & w & 0xaaaaaaaau);
            }
            if (brk) { open = false; par = (uint32_t)(31 - __clz(brk)) & 1u; }
        }
    }
    if (lane == 0) {
        unsigned long long v = 0;
#pragma unroll
        for (int k = 5; k >= 0; --k) v = (v << 10) | f[k];
        seg[q] = v | ((unsigned long long)!open << 60) | ((unsigned long long)par << 61);
    }
}

struct Aff { uint32_t a, c; };
__device__ __forceinline__ Aff aff_mul(Aff g, Aff f) { return Aff{g.a * f.a, g.a * f.c + g.c}; }   // g after f
__device__ __forceinline__ uint32_t lcg_jump(uint32_t s, unsigned long long k) {
    Aff r{1u, 0u}, p{1664525u, 1013904223u};
    while (k) {
        if (k & 1ull) r = aff_mul(p, r);
        p = aff_mul(p, p);
        k >>= 1;
    }
    return r.a * s + r.c;
}

// parity of the run that is open where segment k begins; `known` (>= 0) holds at segment `from`
__device__ uint32_t run_parity(const unsigned long long* seg, long long k, long long from, uint32_t known) {
    while (--k >= from) {
        const unsigned long long v = seg[k];
        if ((v >> 60) & 1ull) return (uint32_t)(v >> 61) & 1u;
    }
    return known;
}

// the draws of each segment's list, in order; block b takes segments [b per, (b + 1) per)
constexpr int DB = 256;
__global__ void __launch_bounds__(DB) k_draw(const uint32_t* list, const unsigned long long* seg, uint32_t nseg, uint32_t per,
                                             uint32_t s0, double p, uint32_t n_bp, uint32_t* hits_words,
                                             unsigned long long* cnt) {
    __shared__ unsigned long long s_sum[DB / 32], s_cand;
    __shared__ int s_last;
    const int lane = threadIdx.x & 31, wl = threadIdx.x >> 5;
    const uint32_t lo = blockIdx.x * per, hi = min(lo + per, nseg);
    if (threadIdx.x == 0) { s_last = -1; s_cand = 0; }
    __syncthreads();
    // draws before the block's first segment, and the last run start before it
    unsigned long long sum = 0;
    int mine = -1;
    for (uint32_t k = threadIdx.x; k < lo; k += DB) {
        const unsigned long long v = seg[k];
        const uint32_t d0 = fld(v, 1), d1 = fld(v, 2);
        sum += fld(v, 0) + (d0 == d1 ? d0 : run_parity(seg, k, 0, 0u) ? d1 : d0);
        if ((v >> 60) & 1ull) mine = (int)k;
    }
    for (int o = 16; o; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if (mine >= 0) atomicMax(&s_last, mine);
    if (lane == 0) s_sum[wl] = sum;
    __syncthreads();
    unsigned long long base = 0;
    for (int k = 0; k < DB / 32; ++k) base += s_sum[k];
    const uint32_t known = s_last >= 0 ? (uint32_t)(seg[s_last] >> 61) & 1u : 0u;
    unsigned long long cand = 0;
    for (uint32_t c = lo; c < hi; c += DB) {
        const uint32_t k = c + threadIdx.x;
        const unsigned long long v = k < hi ? seg[k] : 0ull;
        const uint32_t nres = fld(v, 0), d0 = fld(v, 1), d1 = fld(v, 2), c0 = fld(v, 4), c1 = fld(v, 5);
        const uint32_t par = (d0 | d1 | c0 | c1) ? run_parity(seg, k, lo, known) : 0u;
        cand += fld(v, 3) + (par ? c1 : c0);
        const uint32_t mydraws = nres + (par ? d1 : d0);
        uint32_t off = mydraws;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) { const uint32_t u = __shfl_up_sync(0xffffffffu, off, o); if (lane >= o) off += u; }
        __syncthreads();
        if (lane == 31) s_sum[wl] = off;
        __syncthreads();
        unsigned long long before = base + off - mydraws;
        for (int q = 0; q < DB / 32; ++q) { if (q < wl) before += s_sum[q]; base += s_sum[q]; }
        if (!mydraws) continue;
        uint32_t s = lcg_jump(s0, before);
        for (uint32_t q = 0; q < nres + d0 + d1; ++q) {
            const uint32_t w = list[(unsigned long long)k * SEG + q];
            if ((w >> 31) && ((w >> 30) & 1u) != par) continue;
            s = 1664525u * s + 1013904223u;
            if (s / 4294967296.0 < p) {
                const uint32_t h = w & 0x1fffffffu, shift = (h & 3u) * 8u;
                const uint32_t old = atomicOr(&hits_words[h >> 2], 1u << shift);
                if (((old >> shift) & 0xffu) == 0u) {
                    atomicAdd(&cnt[0], 1ull);
                    atomicAdd(&cnt[h >= n_bp ? 2 : 1], 1ull);
                }
            }
        }
    }
    if (cand) atomicAdd(&s_cand, cand);
    __syncthreads();
    if (threadIdx.x == 0) {
        if (s_cand) atomicAdd(&cnt[3], s_cand);
        if (hi == nseg) cnt[4] = base;
    }
}

// clusterDSB, one block per fibre.  Each thread looks through a run of aligned
// words of either strand (most are zero), counts its hits, and writes them at
// its place in the strand's list: two passes and one scan, where 256 bytes at a
// time with a scan each took three barriers per step (38 us on 441 fibres of 8823
// bp, 7.4 us now).
constexpr int CB = 256;
__global__ void __launch_bounds__(CB) k_cluster(const uint8_t* hits, uint32_t n_per, uint32_t n_bp, uint32_t* out /*3 per fibre*/) {
    extern __shared__ uint32_t lists[];
    __shared__ uint32_t tot[2][CB / 32];
    const int lane = threadIdx.x & 31, wl = threadIdx.x >> 5;
    uint32_t k01[2];
#pragma unroll
    for (int st = 0; st < 2; ++st) {
        const unsigned long long h0 = (unsigned long long)blockIdx.x * n_per + (st ? n_bp : 0u), h1 = h0 + n_per;
        const uint32_t nw = (uint32_t)((h1 + 3) / 4 - h0 / 4), per = (nw + CB - 1) / CB;
        const uint32_t* W = reinterpret_cast<const uint32_t*>(hits) + h0 / 4;
        const uint32_t w0 = min(threadIdx.x * per, nw), w1 = min(w0 + per, nw);
        // bytes equal to 1 inside the fibre, as flags in bit 0 of each byte
        auto ones = [&](uint32_t w) -> uint32_t {
            const uint32_t v = W[w];
            if (v == 0u) return 0u;
            uint32_t m = 0;
            for (int b = 0; b < 4; ++b) {
                const unsigned long long at = (h0 / 4 + w) * 4 + b;
                if (((v >> (8 * b)) & 0xffu) == 1u && at >= h0 && at < h1) m |= 1u << (8 * b);
            }
            return m;
        };
        uint32_t c = 0;
        for (uint32_t w = w0; w < w1; ++w) c += __popc(ones(w));
        uint32_t off = c;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) { const uint32_t u = __shfl_up_sync(0xffffffffu, off, o); if (lane >= o) off += u; }
        if (lane == 31) tot[st][wl] = off;
        __syncthreads();
        uint32_t all = 0;
        off -= c;
        for (int q = 0; q < CB / 32; ++q) { if (q < wl) off += tot[st][q]; all += tot[st][q]; }
        k01[st] = all;
        uint32_t* L = lists + (st ? n_per : 0u);
        if (c)
            for (uint32_t w = w0; w < w1; ++w)
                for (uint32_t m = ones(w); m; m &= m - 1)
                    L[off++] = (uint32_t)((h0 / 4 + w) * 4 + (__ffs(m) - 1) / 8 - h0);
    }
    __syncthreads();
    const uint32_t* s0 = lists;
    const uint32_t k0 = k01[0], k1 = k01[1];
    uint32_t* s1 = lists + n_per;
    if (threadIdx.x == 0) {
        const int W = 10;
        uint32_t dsb = 0, jlo = 0;
        // used flags packed in the high bit of s1 entries
        for (uint32_t a = 0; a < k0; ++a) {
            long long b0 = s0[a];
            while (jlo < k1 && (long long)(s1[jlo] & 0x7fffffffu) < b0 - W) jlo++;
            for (uint32_t j = jlo; j < k1 && (long long)(s1[j] & 0x7fffffffu) <= b0 + W; ++j) {
                if (!(s1[j] >> 31)) { s1[j] |= 0x80000000u; dsb++; break; }
            }
        }
        out[3 * blockIdx.x] = dsb;
        out[3 * blockIdx.x + 1] = k0;
        out[3 * blockIdx.x + 2] = k1;
    }
}

// ------------------------------------------------------------------ host side

cudaError_t launch_score(const float4* rad, const uint32_t* alive, unsigned long long n, const DnaDev& d,
                         double r_d, double p, int dedupe, uint32_t s0, uint32_t* hits_words,
                         const ScoreScratch& sc, cudaStream_t s) {
    if (n == 0) return cudaMemsetAsync(sc.u64, 0, 8 * sizeof(unsigned long long), s);
    const uint32_t nseg = (uint32_t)((n + SEG - 1) / SEG);
    // k_find clears the result counters
    k_find<<<(nseg + FB / 32 - 1) / (FB / 32), FB, 0, s>>>(rad, alive, n, d, r_d, dedupe, sc.list, sc.seg, sc.u64);
    // at least 64 segments to a block: each block reads all summaries before its own
    const uint32_t nb = min((nseg + 63) / 64, 148u), per = (nseg + nb - 1) / nb;
    k_draw<<<(nseg + per - 1) / per, DB, 0, s>>>(sc.list, sc.seg, nseg, per, s0, p, d.n_bp, hits_words, sc.u64);
    return cudaGetLastError();
}

cudaError_t launch_cluster(const uint8_t* hits, const DnaDev& d, uint32_t n_fibers, uint32_t* out, cudaStream_t s) {
    size_t sm = (size_t)d.n_bp_per * 8;
    static DeviceOnce attr;
    cudaError_t e = attr.run([] {
        return cudaFuncSetAttribute(k_cluster, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    });
    if (e != cudaSuccess) return e;
    k_cluster<<<n_fibers, CB, sm, s>>>(hits, d.n_bp_per, d.n_bp, out);
    return cudaGetLastError();
}

uint32_t lcg_jump_host(uint32_t s, unsigned long long k) {
    uint32_t ra = 1u, rc = 0u, pa = 1664525u, pc = 1013904223u;
    while (k) {
        if (k & 1ull) { uint32_t na = pa * ra, nc = pa * rc + pc; ra = na; rc = nc; }
        uint32_t na = pa * pa, nc = pa * pc + pc; pa = na; pc = nc;
        k >>= 1;
    }
    return ra * s + rc;
}

}  // namespace wg
