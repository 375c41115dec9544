// transport.cu -- electron track transport in liquid water (Phase A + B).
//
// Physics follows allaunthefox/webgpu-dna src/shaders/helpers.wgsl:15-186,
// primary.wgsl:41-663 and secondary.wgsl:17-450 (same statements, same f32
// evaluation order); the execution model is new:
//
// * One persistent kernel runs primaries and secondaries together.  A CTA holds
//   256 electrons in shared memory and advances each by one step per iteration
//   (the reference's Phase A loop body for a primary, one Phase B dispatch for a
//   secondary), in phases with a barrier between them: move, then the
//   interactions sorted by kind, then the spurs sorted by kind.  So a warp's
//   lanes run the same branch, the branches of one step run side by side on
//   different warps, and the warps of a CTA fetch the same code.
//   Slots whose electron ended refill from the CTA's stash of secondaries,
//   the global queue or the primary pool, so the reference's 2000 Phase B
//   dispatches become per-secondary step caps.
// * Every particle owns a Philox4x32-10 stream: key = seed, counter =
//   (block, secondary index, primary id, 1).  Results do not depend on which
//   lane or SM runs a particle, or when.
// * rad_buf entries are staged per CTA in shared memory and written out in
//   coalesced bursts with one global atomic per burst; each carries a 64-bit
//   key (pid << 34 | secondary index << 17 | sequence) from which
//   canonicalise() rebuilds a deterministic order.
// * Counters live in shared memory per block; per-lane f64 energy sums.
//
// Compiled with -fmad=false: the only fused multiply-adds are explicit ones.
#include "transport.cuh"
#include "dmath.cuh"

namespace wg {

constexpr int TB = 256;            // threads and electron slots per block
constexpr int TW = TB / 32;        // warps per block
constexpr int STG_FLUSH = 256;     // staged rad entries written out at this level: + 3 per slot and
constexpr int STG = STG_FLUSH + 3 * TB;   // iteration at most
constexpr int STASH = TW * (int)TRANSPORT_STASH / 2;   // secondaries a block keeps in shared memory
constexpr int NREC = 512;          // steps drawn ahead per iteration (few electrons)
constexpr int SHARE = 8;           // secondaries a block gives away per iteration while others have no work
constexpr int QTAKE = 64;          // and takes from the queue at a time

__device__ __forceinline__ unsigned long long gtime() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}


__constant__ float c_SB[5] = {10.79f, 13.39f, 16.05f, 32.30f, 539.0f};
__constant__ float c_EX[5] = {8.22f, 10.00f, 11.24f, 12.61f, 13.77f};
__constant__ float c_DEA_E[14] = {0.0f, 4.2f, 4.3f, 5.8f, 6.0f, 6.2f, 6.4f, 7.0f, 7.5f, 7.7f,
                                  8.4f, 10.2f, 11.2f, 12.3f};
__constant__ float c_DEA_S[14] = {0.0f, 0.0f, 0.0f, 2.5e-5f, 2.8e-4f, 6.0e-4f, 6.7e-4f, 3.7e-4f,
                                  1.09e-4f, 7.0e-5f, 1.4e-4f, 2.0e-5f, 6.0e-5f, 0.0f};
constexpr float NWf = 33.4f;
constexpr float TWO_PI_F = 6.28318530f;
constexpr float PI_F = 3.14159265f;

// counters inside the block's shared block: [0..7] counters, [8..15] sec_stats, [16..23] dbg
enum { C_OH = 0, C_EAQ = 1, C_H = 2, C_H3O = 3, C_DNA = 4, C_H2 = 5,
       SS_CUT = 9, SS_BOUNDS = 10, SS_STEPS = 11, SS_TERT = 12,
       D_IONS = 16, D_EXC = 17, D_ESC = 18, D_PRIM = 19, D_WSUM = 20, D_DOSE = 21 };

// Electron slots, one array per field.  A primary has secondary index 0.
struct Slots {
    float px[TB], py[TB], pz[TB], E[TB], dx[TB], dy[TB], dz[TB];
    uint32_t pid[TB], sub[TB], seq[TB], it[TB];
    uint32_t nd[TB];               // draws taken from its stream
    float tpath[TB], ppath[TB], maxr[TB], sx[TB], sy[TB], sz[TB];   // primaries
    uint32_t nion[TB], nexc[TB], nsec[TB];
    float a[TB], b[TB];            // move -> interaction: table position, flags; ionisation -> spur: W_sec, binding
    float xi[TB], xic[TB], xicv[TB], xicvd[TB], stot[TB], lam[TB], fE[TB];   // cross sections (XS)
    uint32_t iE[TB];
};
// a step drawn ahead: path length, elastic and azimuthal deflection, kind of interaction
struct StepRec { float dist[NREC], ce[NREC], se[NREC], sp[NREC], cp[NREC]; int kind[NREC]; };
enum { L_ION = 0, L_EXC = 1, L_VIB = 2, L_TRACKED = 3, L_SPUR = 4, L_MOVE = 5, NLIST = 6 };

struct Blk {
    const float* T;       // tables
    Slots* S;
    StepRec* R;
    float4* srad;         // rad_buf staging
    unsigned long long* skey;
    int* sn;
    uint32_t* cnt;        // block counters
    StashRec* stash;      // secondaries
    int* stn;
    uint16_t (*list)[TB]; // slots by kind (spurs: | kind << 8)
    uint32_t* ln;         // this iteration's list lengths
};

// One out-of-line copy each of the step's f32 log, exp, pow and sincos: the
// kernel is bound by instruction fetch, and a call is cheaper than another
// inlined copy of the function at every call site.
__device__ __noinline__ float logf_nc(float x) { return logf_pos(x); }
__device__ __noinline__ float expf_nc(float x) { return expf_(x); }
__device__ __noinline__ float powf_nc(float x, float y) { return powf_(x, y); }
__device__ __noinline__ float2 sincosf_nc(float x) { float s, c; sincosf_(x, &s, &c); return make_float2(s, c); }

// Four draws of an electron's stream from draw nd on: the two Philox blocks they can
// lie in, whatever the position in the first, so that the lanes of a warp generate
// together (a draw at a time, some lane needed a new block at nearly every one) and
// nothing but the count is kept between phases.
__device__ __forceinline__ float4 draw4_of(const u4& a, const u4& b, uint32_t ri) {
    const uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
    uint32_t v[6];
#pragma unroll
    for (int k = 0; k < 6; ++k) v[k] = (ri & 1u) ? w[k + 1] : w[k];
    return make_float4(u01f((ri & 2u) ? v[2] : v[0]), u01f((ri & 2u) ? v[3] : v[1]), u01f((ri & 2u) ? v[4] : v[2]),
                       u01f((ri & 2u) ? v[5] : v[3]));
}
// out of line: one copy for all call sites of the interactions and spurs
__device__ __noinline__ float4 draw4_nc(uint32_t nd, uint32_t sub, uint32_t pid, uint32_t k0, uint32_t k1) {
    return draw4_of(philox(nd >> 2, sub, pid, 1u, k0, k1), philox((nd >> 2) + 1u, sub, pid, 1u, k0, k1), nd & 3u);
}

// An electron's stream during a phase.
struct Stream {
    uint32_t nd, sub, pid;
    __device__ __forceinline__ void load(const Slots& S, int s) { nd = S.nd[s]; sub = S.sub[s]; pid = S.pid[s]; }
    __device__ __forceinline__ void store(Slots& S, int s) const { S.nd[s] = nd; }
    // the next four draws; d of them are taken by nd += d
    __device__ __forceinline__ float4 peek(const TArgs& A) const { return draw4_nc(nd, sub, pid, A.k0, A.k1); }
};

__device__ __forceinline__ void put(const TArgs& A, Blk& b, const Stream& q, uint32_t& seq, float x, float y, float z,
                                    float code) {
    int s = atomicAdd(b.sn, 1);
    b.srad[s] = make_float4(x, y, z, code + __uint2float_rn(q.pid) * 8.0f);
    if (seq >= (1u << 17)) atomicOr(&A.st->err, DERR_KEY_RANGE);
    b.skey[s] = ((unsigned long long)(q.pid - A.pid_base) << 34) | ((unsigned long long)q.sub << 17) | seq;
    seq++;
}

// per-thread deposited energy and number of dose-grid atomics
struct Dep { double e; uint32_t n; };

// voxel of (px, py, pz) in the vc^3 dose grid over +-box, or ~0u outside (out of line: 9 call sites)
__device__ __noinline__ uint32_t dose_voxel(float px, float py, float pz, float box, uint32_t vc) {
    float vs = 2.0f * box / (float)vc;
    int ix = (int)floorf((px + box) / vs);
    int iy = (int)floorf((py + box) / vs);
    int iz = (int)floorf((pz + box) / vs);
    int n = (int)vc;
    if (ix < 0 || ix >= n || iy < 0 || iy >= n || iz < 0 || iz >= n) return ~0u;
    return (uint32_t)((iz * n + iy) * n + ix);
}

__device__ __forceinline__ void deposit(const TArgs& A, Dep& dep, float px, float py, float pz, float d) {
    if (d <= 0.0f) return;                                       // primary.wgsl:103
    dep.e += (double)d;
    uint32_t v = dose_voxel(px, py, pz, A.box, A.vc);
    if (v == ~0u) return;
    atomicAdd(&A.dose[v], (uint32_t)(d * 100.0f));
    dep.n++;
}

// dna_near (primary.wgsl:41-86), out of line (4 call sites)
__device__ __noinline__ uint32_t dna_near_nc(float px, float py, float pz, uint32_t N, float spacing, float x0,
                                             float rise, float r_bb);

__device__ __forceinline__ uint32_t dna_near(const TArgs& A, float px, float py, float pz) {
    if (A.dna_enable == 0u) return 0u;
    return dna_near_nc(px, py, pz, A.dna_grid_n, A.dna_spacing, A.dna_x0, A.dna_rise, A.dna_r_bb);
}

__device__ __noinline__ uint32_t dna_near_nc(float px, float py, float pz, uint32_t N, float spacing, float x0,
                                             float rise, float r_bb) {
    const float r_damage = 0.29f;
    float grid_off = -((float)(N - 1u) * spacing) * 0.5f;
    float inv_s = 1.0f / spacing;
    int fi = (int)rintf((py - grid_off) * inv_s);
    int fj = (int)rintf((pz - grid_off) * inv_s);
    if (fi < 0 || fi >= (int)N || fj < 0 || fj >= (int)N) return 0u;
    float fy = grid_off + (float)fi * spacing;
    float fz = grid_off + (float)fj * spacing;
    float y_rel = py - fy, z_rel = pz - fz;
    float r2 = y_rel * y_rel + z_rel * z_rel;
    float R_reach = r_bb + r_damage;
    if (r2 > R_reach * R_reach) return 0u;
    int bp_est = (int)rintf((px - x0) / rise);
    int b0 = bp_est - 1 > 0 ? bp_est - 1 : 0;
    int b1 = bp_est + 1;
    const float d_phase = (float)(2.0 * 3.14159265 / 10.5);
    for (int bb = b0; bb <= b1; ++bb) {
        float bx = x0 + (float)bb * rise;
        float phi = (float)bb * d_phase;
        float s0z, s0y;
        sincosf_(phi, &s0z, &s0y);
        s0y = r_bb * s0y; s0z = r_bb * s0z;
        float dx = px - bx;
        float dy0 = y_rel - s0y, dz0 = z_rel - s0z;
        if (dx * dx + dy0 * dy0 + dz0 * dz0 < r_damage * r_damage) return 1u;
        float s1z, s1y;
        sincosf_(phi + PI_F, &s1z, &s1y);
        s1y = r_bb * s1y; s1z = r_bb * s1z;
        float dy1 = y_rel - s1y, dz1 = z_rel - s1z;
        if (dx * dx + dy1 * dy1 + dz1 * dz1 < r_damage * r_damage) return 1u;
    }
    return 0u;
}

__device__ __forceinline__ float meesungnoen_sigma(float k) {   // primary.wgsl:90-98
    if (k <= 0.1f) return 0.0f;
    float r = -4.06217193e-08f;
    r = r * k + 3.06848412e-06f; r = r * k - 9.93217814e-05f; r = r * k + 1.80172797e-03f;
    r = r * k - 2.01135480e-02f; r = r * k + 1.42939448e-01f; r = r * k - 6.48348714e-01f;
    r = r * k + 1.85227848e+00f; r = r * k - 3.36450378e+00f; r = r * k + 4.37785068e+00f;
    r = r * k - 4.20557339e+00f; r = r * k + 3.81679083e+00f; r = r * k - 2.34069784e-01f;
    return fmaxf(r, 0.0f) * 0.6267f;
}

// Gaussian 3-D displacement from four draws, the mu1..mu4 pattern of primary.wgsl:216-220
__device__ __noinline__ float3 gauss3_nc(float u0, float u1, float u2, float u3, float sigma) {
    const float rr = sqrtf(-2.0f * logf_pos(fmaxf(u0, 1e-30f))) * sigma;
    float sn, cs;
    sincosf_(TWO_PI_F * u1, &sn, &cs);
    const float z = sqrtf(-2.0f * logf_pos(fmaxf(u2, 1e-30f))) * sigma * cosf_(TWO_PI_F * u3);
    return make_float3(rr * cs, rr * sn, z);
}
__device__ __forceinline__ float3 gauss3(const TArgs& A, Stream& q, float sigma) {
    const float4 p = q.peek(A);
    q.nd += 4u;
    return gauss3_nc(p.x, p.y, p.z, p.w, sigma);
}

// H2O+ + eaq -> H2Ovib dissociation channels (primary.wgsl:246-276)
__device__ __forceinline__ void h2ovib(const TArgs& A, Blk& b, const Stream& q, uint32_t& seq, float r_vd, float x, float y,
                                       float z) {
    if (r_vd < 0.1365f) {
        atomicAdd(&b.cnt[C_OH], 2u); atomicAdd(&b.cnt[C_H2], 1u);
        put(A, b, q, seq, x, y, z, 0.0f); put(A, b, q, seq, x, y, z, 0.0f); put(A, b, q, seq, x, y, z, 7.0f);
    } else if (r_vd < 0.494f) {
        atomicAdd(&b.cnt[C_OH], 1u); atomicAdd(&b.cnt[C_H], 1u);
        put(A, b, q, seq, x, y, z, 0.0f); put(A, b, q, seq, x, y, z, 2.0f);
    } else if (r_vd < 0.650f) {
        atomicAdd(&b.cnt[C_H], 2u);
        put(A, b, q, seq, x, y, z, 2.0f); put(A, b, q, seq, x, y, z, 2.0f);
    }
}

__device__ __forceinline__ void rotate(float& dx, float& dy, float& dz, float ct, float st, float cp, float sp) {
    if (fabsf(dz) > 0.99999f) {                                  // primary.wgsl:169-170
        float sw = (dz > 0.0f) ? 1.0f : -1.0f;
        dx = st * cp; dy = st * sp * sw; dz = ct * sw;
    } else {
        float qq = sqrtf(1.0f - dz * dz);
        float inv = 1.0f / qq;
        float nx = dx * ct + st * (dx * dz * cp - dy * sp) * inv;
        float ny = dy * ct + st * (dy * dz * cp + dx * sp) * inv;
        float nz = dz * ct - qq * st * cp;
        float len = sqrtf(nx * nx + ny * ny + nz * nz);
        dx = nx / len; dy = ny / len; dz = nz / len;
    }
}

// Born differential CDF: the reference scans breakpoints linearly
// (helpers.wgsl:98-105) for the last j in [0, N_WR-2] whose prefix is <= r.
// Every committed CDF row is non-decreasing, so the index is
// (number of breakpoints <= r) - 1: a guide table in shared memory (every 16th
// breakpoint) picks the 16-wide window, whose (CDF, energy) pairs are then
// fetched together with independent loads.
__device__ __forceinline__ float sample_W_sec(const TArgs& A, const float* T, float E, uint32_t shell, float r) {
    uint32_t lo = 0, hi = NWE_ - 1;                              // helpers.wgsl:88-96
    while (hi - lo > 1u) { uint32_t mid = (lo + hi) / 2u; if (T[S_XWE + mid] <= E) lo = mid; else hi = mid; }
    uint32_t iE = (fabsf(T[S_XWE + hi] - E) < fabsf(T[S_XWE + lo] - E)) ? hi : lo;
    const float* G = T + S_GUIDE + (shell * NWE_ + iE) * GUIDES;
    int M = 0;
#pragma unroll
    for (int m = 0; m < GUIDES; ++m) M += (G[m] <= r) ? 1 : 0;
    int base = 16 * (M - 1);
    const float2* row = A.tab.xcw + (size_t)(shell * NWE_ + iE) * NWR_;
    int cnt = 0;
#pragma unroll
    for (int k = 1; k <= 16; ++k) {
        int idx = base + k;
        if (idx <= NWR_ - 2) cnt += (__ldg(row + idx).x <= r) ? 1 : 0;
    }
    uint32_t jlo = (uint32_t)(base + cnt);
    uint32_t jhi = jlo + 1 < NWR_ - 1 ? jlo + 1 : NWR_ - 1;
    float2 a = __ldg(row + jlo), b = __ldg(row + jhi);
    float c0 = a.x, c1 = b.x, e0 = a.y, e1 = b.y;
    if (c1 <= c0) return e0;
    float f = fminf(fmaxf((r - c0) / (c1 - c0), 0.0f), 1.0f);
    return e0 + (e1 - e0) * f;
}

// Write one record to the global queue; the consumer spins on the epoch flag
// written after the payload.  Records beyond the queue capacity are dropped and
// counted, as sec_dropped in the reference.
__device__ __forceinline__ void push_global(const TArgs& A, unsigned long long slot, const StashRec& r) {
    if (slot >= A.max_sec) { atomicAdd(&A.st->sec_drop, 1u); return; }
    SecRec* rec = A.secq + slot;
    rec->pe = make_float4(r.x, r.y, r.z, r.E);
    rec->dir = make_float4(r.dx, r.dy, r.dz, 0.0f);
    rec->meta.x = r.pid;
    rec->meta.y = r.sub;
    __threadfence();
    *(volatile uint32_t*)&rec->meta.z = A.pub_epoch;     // publish
}

// the lanes of the warp with `on` append their slot to a list; their place in it
__device__ __forceinline__ int push_list(Blk& b, int k, bool on, uint32_t v, int lane) {
    const unsigned m = __ballot_sync(0xffffffffu, on);
    if (!m) return 0;
    uint32_t base = 0;
    if (lane == __ffs(m) - 1) base = atomicAdd(&b.ln[k], (uint32_t)__popc(m));
    base = __shfl_sync(0xffffffffu, base, __ffs(m) - 1);
    base += __popc(m & ((1u << lane) - 1u));
    if (on) b.list[k][base] = (uint16_t)v;
    return (int)base;
}

// Spurs: an ionisation whose e-aq thermalises nearby (code 5, displaced from the
// ionisation site), a primary's ionisation with a tracked secondary (separation
// estimated from the secondary's range, no e-aq entry; its own list), an
// autoionising excitation (code 1, e-aq displaced from the displaced mother
// site), and a secondary that thermalises below the cutoff (its e-aq alone, code
// 5, secondary.wgsl:100-124).
enum : int { SPUR_NONE = 0, SPUR_LOCAL = 1, SPUR_TRACKED = 2, SPUR_AUTO = 3, SPUR_THERM = 4 };

// ---- interactions after the move (primary.wgsl:180-649, secondary.wgsl:167-443);
// every electron draws in the reference's statement order.

// ionisation; returns the spur it starts
__device__ __forceinline__ int ionise(const TArgs& A, Blk& b, int s, Dep& dep) {
    const float* T = b.T;
    Slots& S = *b.S;
    Stream q;
    q.load(S, s);
    float E = S.E[s];
    const float px = S.px[s], py = S.py[s], pz = S.pz[s], t = S.a[s];
    const int grid = (int)(__float_as_uint(S.b[s]) & 3u) - 1;
    const bool prim = q.sub == 0u;
    const float4 d = q.peek(A);
    float sf[5];
    if (grid < 0) { for (int k = 0; k < 5; ++k) sf[k] = T[S_XSF + k * XN_]; }
    else if (grid > 0) { for (int k = 0; k < 5; ++k) sf[k] = T[S_XSF + k * XN_ + XN_ - 1]; }
    else {
        uint32_t i = (uint32_t)fminf(fmaxf(floorf(t), 0.0f), (float)(XN_ - 2));
        float f = t - (float)i;
        for (int k = 0; k < 5; ++k) {
            const float* a = T + S_XSF + k * XN_;
            sf[k] = fmaxf(0.0f, a[i] + (a[i + 1] - a[i]) * f);
        }
    }
    float fsum = fmaxf(sf[0] + sf[1] + sf[2] + sf[3] + sf[4], 1e-12f);
    float r_sh = d.x * fsum;
    uint32_t shell;
    float bind;
    if (r_sh < sf[0]) { bind = c_SB[0]; shell = 0; }
    else if (r_sh < sf[0] + sf[1]) { bind = c_SB[1]; shell = 1; }
    else if (r_sh < sf[0] + sf[1] + sf[2]) { bind = c_SB[2]; shell = 2; }
    else if (r_sh < sf[0] + sf[1] + sf[2] + sf[3]) { bind = c_SB[3]; shell = 3; }
    else { bind = c_SB[4]; shell = 4; }
    if (!(E > bind)) {
        S.nd[s] = q.nd + 1u;
        return SPUR_NONE;
    }
    S.nd[s] = q.nd + 2u;
    float Wmax = (E + bind) * 0.5f;
    float W = sample_W_sec(A, T, E, shell, d.y);
    W = fminf(fmaxf(W, bind), Wmax);
    const float W_sec = fmaxf(W - bind, 0.0f);
    E -= W;
    if (prim) {
        S.nion[s]++;
        atomicAdd(&b.cnt[D_WSUM], (uint32_t)(W * 10.0f));
        deposit(A, dep, px, py, pz, bind);
        if (W_sec <= A.ce) deposit(A, dep, px, py, pz, W_sec);
    } else {                                             // secondary.wgsl:192-255
        atomicAdd(&b.cnt[SS_TERT], 1u);
        deposit(A, dep, px, py, pz, W);
    }
    if (dna_near(A, px, py, pz) == 1u) atomicAdd(&b.cnt[C_DNA], 1u);
    S.E[s] = E;
    S.a[s] = W_sec;
    S.b[s] = bind;
    return (!prim || W_sec <= A.ce) ? SPUR_LOCAL : SPUR_TRACKED;
}

// excitation; returns the spur it starts
__device__ __forceinline__ int excite(const TArgs& A, Blk& b, int s, Dep& dep) {
    const float* T = b.T;
    Slots& S = *b.S;
    Stream q;
    q.load(S, s);
    const float E = S.E[s], px = S.px[s], py = S.py[s], pz = S.pz[s], t = S.a[s];
    const int grid = (int)(__float_as_uint(S.b[s]) & 3u) - 1;
    const float4 p = q.peek(A);
    S.nd[s] = q.nd + 2u;
    float ef[5];
    if (grid < 0) { for (int k = 0; k < 5; ++k) ef[k] = T[S_XEF + k * XN_]; }
    else if (grid > 0) { for (int k = 0; k < 5; ++k) ef[k] = T[S_XEF + k * XN_ + 85]; }
    else {
        uint32_t i = (uint32_t)fminf(fmaxf(floorf(t), 0.0f), (float)(XN_ - 2));
        if (i > 85u) i = 85u;
        float f = (i == 85u) ? 0.0f : t - (float)i;
        uint32_t j = i + 1 < 85u ? i + 1 : 85u;
        for (int k = 0; k < 5; ++k) {
            const float* a = T + S_XEF + k * XN_;
            ef[k] = fmaxf(0.0f, a[i] + (a[j] - a[i]) * f);
        }
    }
    float efsum = fmaxf(ef[0] + ef[1] + ef[2] + ef[3] + ef[4], 1e-12f);
    float r_ex = p.x * efsum;
    float exc_E; uint32_t lvl;
    if (r_ex < ef[0]) { exc_E = c_EX[0]; lvl = 0; }
    else if (r_ex < ef[0] + ef[1]) { exc_E = c_EX[1]; lvl = 1; }
    else if (r_ex < ef[0] + ef[1] + ef[2]) { exc_E = c_EX[2]; lvl = 2; }
    else if (r_ex < ef[0] + ef[1] + ef[2] + ef[3]) { exc_E = c_EX[3]; lvl = 3; }
    else { exc_E = c_EX[4]; lvl = 4; }
    float d = fminf(exc_E, E);
    S.E[s] = E - d;
    deposit(A, dep, px, py, pz, d);
    if (q.sub == 0u) S.nexc[s]++;
    const float r_ch = p.y;
    int spur = SPUR_NONE;
    // channel: 1 OH + H, 2 2 OH + H2, 3 2 H
    int ch = 0;
    if (lvl == 0u) {
        if (r_ch < 0.65f) ch = 1;
    } else if (lvl == 1u) {
        if (r_ch < 0.175f) {
        } else if (r_ch < 0.2075f) ch = 2;
        else if (r_ch < 0.7075f) spur = SPUR_AUTO;           // primary.wgsl:473-536
        else if (r_ch < 0.961f) ch = 1;
        else ch = 3;
    } else {
        if (r_ch < 0.50f) spur = SPUR_AUTO;                  // primary.wgsl:560-619
    }
    if (ch) {
        uint32_t seq = S.seq[s];
        if (ch != 3) put(A, b, q, seq, px, py, pz, 0.0f);
        if (ch == 2) put(A, b, q, seq, px, py, pz, 0.0f);
        if (ch == 2) put(A, b, q, seq, px, py, pz, 7.0f);
        else put(A, b, q, seq, px, py, pz, 2.0f);
        if (ch == 3) put(A, b, q, seq, px, py, pz, 2.0f);
        S.seq[s] = seq;
        if (ch != 3) atomicAdd(&b.cnt[C_OH], (uint32_t)ch);
        if (ch == 2) atomicAdd(&b.cnt[C_H2], 1u);
        else atomicAdd(&b.cnt[C_H], ch == 3 ? 2u : 1u);
    }
    if (dna_near(A, px, py, pz) == 1u) atomicAdd(&b.cnt[C_DNA], 1u);
    return spur;
}

// vibrational excitation, or dissociative attachment
__device__ __forceinline__ void vibrate(const TArgs& A, Blk& b, int s, Dep& dep) {
    const float* T = b.T;
    Slots& S = *b.S;
    Stream q;
    q.load(S, s);
    const float E = S.E[s], px = S.px[s], py = S.py[s], pz = S.pz[s];
    const uint32_t meta = __float_as_uint(S.b[s]);
    if (meta & 4u) {                                             // Melton DEA
        deposit(A, dep, px, py, pz, E);
        atomicAdd(&b.cnt[C_OH], 1u); atomicAdd(&b.cnt[C_H2], 1u);
        uint32_t seq = S.seq[s];
        put(A, b, q, seq, px, py, pz, 0.0f); put(A, b, q, seq, px, py, pz, 6.0f); put(A, b, q, seq, px, py, pz, 7.0f);
        S.seq[s] = seq;
        S.E[s] = 0.0f;
        return;
    }
    // sample_vib_mode (helpers.wgsl:148-170) with the bin found by the move
    const float4 p = q.peek(A);
    S.nd[s] = q.nd + 1u;
    const uint32_t base = (meta >> 3) * 9u;
    float cumsum = 0.0f, cs[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) {
        float frac = (T[S_VIB + k] > E) ? 0.0f : T[S_XVMF + base + k];
        cumsum = cumsum + frac;
        cs[k] = cumsum;
    }
    uint32_t mode = 8u;
    if (cumsum <= 0.0f) mode = 0u;
    else {
        float thr = p.x * cumsum;
#pragma unroll
        for (int k = 8; k >= 0; --k) if (thr < cs[k]) mode = (uint32_t)k;
    }
    float d = fminf(T[S_VIB + mode], E);
    S.E[s] = E - d;
    deposit(A, dep, px, py, pz, d);
}

// ---- spurs: mother (H2O+) displacement, then e-aq displacement and Onsager
// recombination (p = 1 - exp(-0.711 / r)) or the tracked-secondary estimate
// r = 0.04 W^1.3 + meesungnoen(min(W, 7.4)), then the H2Ovib channels or the
// OH + [e-aq] + H3O+ entries (primary.wgsl:216-353)
__device__ __forceinline__ void spur(const TArgs& A, Blk& b, int s, int kind) {
    Slots& S = *b.S;
    Stream q;
    q.load(S, s);
    uint32_t seq = S.seq[s];
    const float px = S.px[s], py = S.py[s], pz = S.pz[s];
    float mpx = px, mpy = py, mpz = pz;
    if (kind != SPUR_THERM) {
        const float3 m = gauss3(A, q, 1.1547005f);
        mpx = px + m.x; mpy = py + m.y; mpz = pz + m.z;
    }
    float epx = px, epy = py, epz = pz;
    if (kind == SPUR_AUTO) { epx = mpx; epy = mpy; epz = mpz; }
    const float eaq_s = meesungnoen_sigma(kind == SPUR_AUTO ? 1.7f : kind == SPUR_THERM ? S.E[s] : S.a[s]);
    if (eaq_s > 0.0f) {
        const float3 g = gauss3(A, q, eaq_s);
        epx = epx + g.x; epy = epy + g.y; epz = epz + g.z;
    }
    if (kind == SPUR_THERM) {
        put(A, b, q, seq, epx, epy, epz, 5.0f);
        return;                                                  // the slot is free
    }
    const float4 p = q.peek(A);
    const float rdx = epx - mpx, rdy = epy - mpy, rdz = epz - mpz;
    const float r_sep = fmaxf(sqrtf(rdx * rdx + rdy * rdy + rdz * rdz), 1e-6f);
    const float p_recomb = 1.0f - expf_nc(-0.711f / r_sep);
    if (p.x < p_recomb) {
        q.nd += 2u;
        h2ovib(A, b, q, seq, p.y, mpx, mpy, mpz);
    } else {
        q.nd += 1u;
        atomicAdd(&b.cnt[C_OH], 1u); atomicAdd(&b.cnt[C_H3O], 1u); atomicAdd(&b.cnt[C_EAQ], 1u);
        put(A, b, q, seq, mpx, mpy, mpz, 0.0f);
        put(A, b, q, seq, epx, epy, epz, kind == SPUR_AUTO ? 1.0f : 5.0f);
        put(A, b, q, seq, mpx, mpy, mpz, 3.0f);
    }
    S.seq[s] = seq;
    q.store(S, s);
}

// the spur of a primary's ionisation above the cutoff, and its secondary
__device__ __forceinline__ void spur_tracked(const TArgs& A, Blk& b, int s, uint32_t sec_idx) {
    Slots& S = *b.S;
    Stream q;
    q.load(S, s);
    uint32_t seq = S.seq[s];
    const float px = S.px[s], py = S.py[s], pz = S.pz[s], W_sec = S.a[s], bind = S.b[s];
    const float3 m = gauss3(A, q, 1.1547005f);
    const float mpx = px + m.x, mpy = py + m.y, mpz = pz + m.z;
    const float r_track = 0.04f * powf_nc(W_sec, 1.3f);
    const float r_tail = meesungnoen_sigma(fminf(W_sec, 7.4f));
    const float r_sep_est = fmaxf(r_track + r_tail, 1e-3f);
    const float p_recomb = 1.0f - expf_nc(-0.711f / r_sep_est);
    {
        const float4 p = q.peek(A);
        if (p.x < p_recomb) {
            q.nd += 2u;
            h2ovib(A, b, q, seq, p.y, mpx, mpy, mpz);
        } else {
            q.nd += 1u;
            atomicAdd(&b.cnt[C_OH], 1u); atomicAdd(&b.cnt[C_H3O], 1u);
            put(A, b, q, seq, mpx, mpy, mpz, 0.0f);
            put(A, b, q, seq, mpx, mpy, mpz, 3.0f);
        }
    }
    S.seq[s] = seq;
    // primary.wgsl:362-413: at or beyond max_sec the secondary is dropped
    // together with its angle draws and the primary's momentum update (:364)
    if (sec_idx < A.max_sec) {
        const uint32_t nsec = S.nsec[s] + 1u;
        S.nsec[s] = nsec;
        const float E_before = S.E[s] + bind + W_sec;
        const float4 p = q.peek(A);
        uint32_t nd = 0;
        float cos_s;
        if (W_sec < 50.0f) {
            cos_s = 2.0f * p.x - 1.0f;
            nd = 1;
        } else if (W_sec <= 200.0f) {
            cos_s = p.x <= 0.1f ? 2.0f * p.y - 1.0f : p.y * 0.70710678f;
            nd = 2;
        } else {
            float sin2 = fminf(fmaxf((1.0f - W_sec / E_before) / (1.0f + W_sec / 1022000.0f), 0.0f), 1.0f);
            cos_s = sqrtf(fmaxf(0.0f, 1.0f - sin2));
        }
        const float sin_s = sqrtf(fmaxf(0.0f, 1.0f - cos_s * cos_s));
        const float2 sc = sincosf_nc(TWO_PI_F * (nd == 0u ? p.x : nd == 1u ? p.y : p.z));
        q.nd += nd + 1u;
        const float qx = S.dx[s], qy = S.dy[s], qz = S.dz[s];
        float sdx = qx, sdy = qy, sdz = qz;
        rotate(sdx, sdy, sdz, cos_s, sin_s, sc.y, sc.x);
        const float p_inc = sqrtf(E_before), p_sec = sqrtf(W_sec);
        const float pfx = p_inc * qx - p_sec * sdx;
        const float pfy = p_inc * qy - p_sec * sdy;
        const float pfz = p_inc * qz - p_sec * sdz;
        const float pfl = sqrtf(pfx * pfx + pfy * pfy + pfz * pfz);
        if (pfl > 1e-10f) { S.dx[s] = pfx / pfl; S.dy[s] = pfy / pfl; S.dz[s] = pfz / pfl; }
        if (nsec >= (1u << 17)) atomicOr(&A.st->err, DERR_KEY_RANGE);
        const StashRec r{px, py, pz, W_sec, sdx, sdy, sdz, q.pid, nsec};
        const int slot = A.stash_spill ? atomicAdd(b.stn, 1) : STASH;
        if (slot < STASH) b.stash[slot] = r;
        else push_global(A, atomicAdd(&A.st->sec_qtail.v, 1u), r);
    }
    q.store(S, s);
}

// ---- cross sections at the electron's energy (helpers.wgsl:15-66, 134-186).  They
// hold until an interaction changes the energy, so a run of elastic steps
// shares them.
struct XS {
    float xi, xic, xicv, xicvd;    // running sums of ionisation, excitation, vibration, attachment
    float s_tot, lambda, fE;       // total, mean free path; place in the elastic table
    uint32_t iE;
    float t;                       // place in the energy grid
    uint32_t meta;                 // grid + 1 | vibrational bin << 3
};
__device__ __forceinline__ bool cross_sections(const TArgs& A, const float* T, float E, XS& x) {
    float xi, xc, xl;
    int grid;
    x.t = 0.0f;
    const float lE = logf_nc(E);
    if (E <= T[S_XE]) { grid = -1; xi = 0.0f; xc = 0.0f; xl = T[S_XL]; }
    else if (E >= T[S_XE + XN_ - 1]) { grid = 1; xi = T[S_XI + XN_ - 1]; xc = T[S_XC + XN_ - 1]; xl = T[S_XL + XN_ - 1]; }
    else {
        grid = 0;
        x.t = (lE - A.tab.log_xe0) * A.tab.inv_log_xe_step;
        uint32_t i = (uint32_t)fminf(fmaxf(floorf(x.t), 0.0f), (float)(XN_ - 2));
        float f = x.t - (float)i;
        xi = fmaxf(0.0f, T[S_XI + i] + (T[S_XI + i + 1] - T[S_XI + i]) * f);
        xc = fmaxf(0.0f, T[S_XC + i] + (T[S_XC + i + 1] - T[S_XC + i]) * f);
        xl = fmaxf(0.0f, T[S_XL + i] + (T[S_XL + i + 1] - T[S_XL + i]) * f);
    }
    float svib = 0.0f;
    uint32_t vbin = 0;
    if (E >= 2.0f && E < 100.0f) {                               // xs_vib_total
        uint32_t lo = 0, hi = NVIB_ - 1;
        while (hi - lo > 1u) { uint32_t mid = (lo + hi) >> 1; if (T[S_XVE + mid] <= E) lo = mid; else hi = mid; }
        vbin = lo;
        float f = (E - T[S_XVE + lo]) / (T[S_XVE + lo + 1] - T[S_XVE + lo]);
        svib = fmaxf(0.0f, T[S_XVS + lo] + (T[S_XVS + lo + 1] - T[S_XVS + lo]) * f);
    }
    float sdea = 0.0f;
    if (E >= 4.0f && E <= 13.0f) {                               // xs_dea
        int i = 0;                                               // last breakpoint <= E
#pragma unroll
        for (int k = 1; k < 14; ++k) i += E >= c_DEA_E[k] ? 1 : 0;
        if (i < 13) {
            float f = (E - c_DEA_E[i]) / (c_DEA_E[i + 1] - c_DEA_E[i]);
            sdea = fmaxf(0.0f, c_DEA_S[i] + (c_DEA_S[i + 1] - c_DEA_S[i]) * f);
        }
    }
    x.s_tot = xi + xc + xl + svib + sdea;
    if (x.s_tot <= 0.0f) return false;
    x.xi = E > c_SB[0] ? xi : -1.0f;                             // no ionisation below the first shell
    x.xic = xi + xc;
    x.xicv = x.xic + svib;
    x.xicvd = x.xicv + sdea;
    x.lambda = 1.0f / (NWf * x.s_tot);
    const float lEa = (E >= T[S_XAE]) ? lE : logf_nc(T[S_XAE]);
    const float tE = (lEa - A.tab.log_xae0) * A.tab.inv_log_xae_step;
    x.iE = (uint32_t)fminf(fmaxf(floorf(tE), 0.0f), (float)(NAE_ - 2));
    x.fE = fminf(fmaxf(tE - (float)x.iE, 0.0f), 1.0f);
    x.meta = (uint32_t)(grid + 1) | (vbin << 3);
    return true;
}

__device__ __forceinline__ void start_primary(const TArgs& A, Slots& S, int s, uint32_t idx) {
    Stream q;
    q.nd = 0; q.sub = 0; q.pid = A.pid_base + idx;
    float px = 0.0f, py = 0.0f, pz = 0.0f;
    const float sh = A.start_half;
    if (sh > 0.0f) {
        const float4 p = q.peek(A);
        q.nd += 3u;
        px = (p.x * 2.0f - 1.0f) * sh;
        py = (p.y * 2.0f - 1.0f) * sh;
        pz = (p.z * 2.0f - 1.0f) * sh;
    }
    const float4 p = q.peek(A);
    q.nd += 2u;
    const float u1 = fmaxf(p.x, 1e-10f);
    const float cos_i = 1.0f - 2.0f * u1;
    const float sin_i = sqrtf(fmaxf(0.0f, 1.0f - cos_i * cos_i));
    float spi, cpi;
    sincosf_(TWO_PI_F * p.y, &spi, &cpi);
    S.px[s] = px; S.py[s] = py; S.pz[s] = pz;
    S.sx[s] = px; S.sy[s] = py; S.sz[s] = pz;
    S.E[s] = A.E_prim ? A.E_prim[idx] : A.be;
    S.dx[s] = sin_i * cpi; S.dy[s] = sin_i * spi; S.dz[s] = cos_i;
    S.pid[s] = q.pid; S.sub[s] = 0; S.seq[s] = 0; S.it[s] = 0; S.nsec[s] = 0;
    S.tpath[s] = 0.0f; S.ppath[s] = 0.0f; S.maxr[s] = 0.0f; S.nion[s] = 0; S.nexc[s] = 0;
    q.store(S, s);
}

__device__ __forceinline__ void load_secondary(Slots& S, int s, const StashRec& r) {
    S.px[s] = r.x; S.py[s] = r.y; S.pz[s] = r.z; S.E[s] = r.E;
    S.dx[s] = r.dx; S.dy[s] = r.dy; S.dz[s] = r.dz;
    S.pid[s] = r.pid; S.sub[s] = r.sub; S.seq[s] = 0; S.it[s] = 0; S.nd[s] = 0;
}

__device__ __forceinline__ void finish_primary(const TArgs& A, Blk& b, int s, Dep& dep, float px, float py, float pz,
                                               uint32_t esc) {
    const Slots& S = *b.S;
    const float E = S.E[s];
    if (esc == 0u && E > 0.0f) deposit(A, dep, px, py, pz, E);
    float4* r = reinterpret_cast<float4*>(A.results + 8ull * (S.pid[s] - A.pid_base));
    r[0] = make_float4(S.tpath[s], S.ppath[s], E, __uint_as_float(S.nion[s]));
    r[1] = make_float4(__uint_as_float(S.nexc[s]), __uint_as_float(esc), S.maxr[s], 0.0f);
    A.nsec[S.pid[s] - A.pid_base] = S.nsec[s];
    atomicAdd(&b.cnt[D_IONS], S.nion[s]); atomicAdd(&b.cnt[D_EXC], S.nexc[s]);
    atomicAdd(&b.cnt[D_ESC], esc); atomicAdd(&b.cnt[D_PRIM], 1u);
}

// ---- the move: steps (primary.wgsl:155-172: free flight, elastic deflection, kind of
// interaction, four draws) until one interacts.  Five of six steps are elastic
// only; they leave the energy and so the cross sections alone, and need no other
// phase, so an iteration takes a run of them.

// a step's draws: all of it that does not depend on where the electron is
struct Step { float dist, ce, se, sp, cp; int kind; };
__device__ __forceinline__ Step draw_step(const float* T, const float4& u, float lambda, uint32_t iE, float fE, float s_tot,
                                          float xi, float xic, float xicv, float xicvd) {
    Step r;
    r.dist = -logf_nc(fmaxf(u.x, 1e-10f)) * lambda;
    // xs_el_cos (helpers.wgsl:66-82)
    const float* a0 = T + S_XAC + iE * NAC_;
    const float* a1 = a0 + NAC_;
    const float rr = fminf(fmaxf(u.y, 0.0f), 1.0f);
    const float jf = rr * (float)(NAC_ - 1);
    const uint32_t jlo = (uint32_t)floorf(jf);
    const uint32_t jhi = jlo + 1 < NAC_ - 1 ? jlo + 1 : NAC_ - 1;
    const float fj = jf - (float)jlo;
    const float cE0 = a0[jlo] + (a0[jhi] - a0[jlo]) * fj;
    const float cE1 = a1[jlo] + (a1[jhi] - a1[jlo]) * fj;
    r.ce = fminf(fmaxf(cE0 + (cE1 - cE0) * fE, -1.0f), 1.0f);
    r.se = sqrtf(fmaxf(0.0f, 1.0f - r.ce * r.ce));
    const float2 sc = sincosf_nc(TWO_PI_F * u.z);
    r.sp = sc.x;
    r.cp = sc.y;
    const float r_type = u.w * s_tot;
    // list | attachment << 8, or -1: elastic only
    r.kind = r_type < xi ? L_ION : r_type < xic ? L_EXC : r_type < xicv ? L_VIB : r_type < xicvd ? L_VIB | 256 : -1;
    return r;
}

// an electron between steps
struct Flight {
    float px, py, pz, dx, dy, dz, tpath, ppath, maxr, sx, sy, sz;
    uint32_t it, it_max, n;
    bool prim, productive;
    __device__ __forceinline__ void load(const Slots& S, int s, const TArgs& A) {
        px = S.px[s]; py = S.py[s]; pz = S.pz[s]; dx = S.dx[s]; dy = S.dy[s]; dz = S.dz[s];
        tpath = S.tpath[s]; ppath = S.ppath[s]; maxr = S.maxr[s]; sx = S.sx[s]; sy = S.sy[s]; sz = S.sz[s];
        it = S.it[s]; n = 0;
        prim = S.sub[s] == 0u;
        productive = S.E[s] > 12.0f;
        it_max = prim ? A.ms : A.sec_steps;
    }
    // takes a step; true: the run ends here (what the step drew, the box, the step cap)
    __device__ __forceinline__ bool step(const Step& r, float box, int& kind, bool& esc) {
        rotate(dx, dy, dz, r.ce, r.se, r.cp, r.sp);
        px += dx * r.dist; py += dy * r.dist; pz += dz * r.dist;
        ++n;
        ++it;
        const bool out = fabsf(px) >= box || fabsf(py) >= box || fabsf(pz) >= box;
        if (prim) {
            tpath += r.dist;
            if (productive) ppath += r.dist;
            const float rdx = px - sx, rdy = py - sy, rdz = pz - sz;
            const float rad = sqrtf(rdx * rdx + rdy * rdy + rdz * rdz);
            if (rad > maxr) maxr = rad;
            if (out) { esc = true; return true; }
        }
        kind = r.kind;
        // a secondary that leaves the box or reaches the cap still interacts
        return kind >= 0 || out || it >= it_max;
    }
    __device__ __forceinline__ void store(Slots& S, int s) const {
        S.px[s] = px; S.py[s] = py; S.pz[s] = pz; S.dx[s] = dx; S.dy[s] = dy; S.dz[s] = dz;
        if (prim) { S.tpath[s] = tpath; S.ppath[s] = ppath; S.maxr[s] = maxr; }
        S.it[s] = it;
    }
};

// What comes before a run of steps: the reference's checks and the cross
// sections.  0: go; 1: ended; 2: thermalised (a spur follows).
__device__ __forceinline__ int begin_move(const TArgs& A, Blk& b, int s, Dep& dep, XS& x) {
    Slots& S = *b.S;
    const float box = A.box, E = S.E[s], px = S.px[s], py = S.py[s], pz = S.pz[s];
    const bool prim = S.sub[s] == 0u;
    const bool capped = S.it[s] >= (prim ? A.ms : A.sec_steps);
    int esc = -1;                                                // a primary's end (1: left the box)
    if (capped || (prim && E < A.ce)) esc = 0;
    else if (E < A.ce) {                                         // secondary.wgsl:100-124
        deposit(A, dep, px, py, pz, E);
        atomicAdd(&b.cnt[C_EAQ], 1u);
        atomicAdd(&b.cnt[SS_CUT], 1u);
        return 2;
    } else if (fabsf(px) >= box || fabsf(py) >= box || fabsf(pz) >= box) {
        if (!prim) atomicAdd(&b.cnt[SS_BOUNDS], 1u);
        esc = 1;
    } else if (!cross_sections(A, b.T, E, x)) esc = 0;
    if (esc < 0) return 0;
    if (prim) finish_primary(A, b, s, dep, px, py, pz, (uint32_t)esc);
    return 1;
}

// What comes after it; the list that follows, or -1
__device__ __forceinline__ int end_move(const TArgs& A, Blk& b, int s, Dep& dep, unsigned long long& nsteps, const Flight& f,
                                        float t, uint32_t meta, int kind, bool esc, bool& active) {
    Slots& S = *b.S;
    nsteps += f.n;
    if (!f.prim) atomicAdd(&b.cnt[SS_STEPS], f.n);
    f.store(S, s);
    S.nd[s] += 4u * f.n;
    if (esc) {
        finish_primary(A, b, s, dep, f.px, f.py, f.pz, 1u);
        active = false;
        return -1;
    }
    S.a[s] = t;
    S.b[s] = __uint_as_float(kind >= 256 ? meta | 4u : meta);
    return kind < 0 ? -1 : kind & 255;
}

// Many electrons: a lane draws and takes its own steps, at most `most` (a warp
// waits for its longest run).  Returns the list that follows (-1: none) and clears
// `active` when the electron ends.
// With secondaries waiting, work is what counts: MOVE_STEPS; else the run's length
// is latency: MOVE_STEPS_FEW.  Measured (ms at 4096 x 10 keV; 4096 x 1 keV; 16,384 of 0.1 to
// 30 keV): 12 and 4 4.51, 1.05, 10.62; 6 and 4 4.48, 1.04, 10.28; 6 and 3 4.35, 1.06,
// 10.20; 5 and 2 4.54, 1.10, 10.17; 12 and 1 5.4, 1.24, 11.6.
constexpr uint32_t MOVE_STEPS = 6, MOVE_STEPS_FEW = 3;
__device__ __forceinline__ int move(const TArgs& A, Blk& b, int s, Dep& dep, unsigned long long& nsteps, bool& active,
                                    uint32_t most) {
    Slots& S = *b.S;
    XS x;
    const int go = begin_move(A, b, s, dep, x);
    if (go) { active = false; return go == 2 ? L_SPUR : -1; }
    Flight f;
    f.load(S, s, A);
    const uint32_t nd = S.nd[s], sub = S.sub[s], pid = S.pid[s];
    u4 cur = philox(nd >> 2, sub, pid, 1u, A.k0, A.k1);
    int kind = -1;
    bool esc = false;
#pragma unroll 1
    for (uint32_t k = 1; k <= most; ++k) {
        const u4 nxt = philox((nd >> 2) + k, sub, pid, 1u, A.k0, A.k1);
        const Step r = draw_step(b.T, draw4_of(cur, nxt, nd & 3u), x.lambda, x.iE, x.fE, x.s_tot, x.xi, x.xic, x.xicv, x.xicvd);
        cur = nxt;
        if (f.step(r, A.box, kind, esc)) break;
    }
    return end_move(A, b, s, dep, nsteps, f, x.t, x.meta, kind, esc, active);
}

// What bounds it: the chain of a primary's steps (650 at 10 keV), each as long as
// an iteration takes.  2 CTAs per SM hold 512 electrons; at 4096 x 10 keV about 325
// are alive at a time, so an iteration costs little more than its longest
// phase path, and with more electrons the issue slots bind.
// Measured at 4096 x 10 keV: 14.9 ms with one warp per 32 electrons taking all
// branches one after another (7.8 lanes per instruction, 16 % issue), 4.5 ms now.
__global__ void __launch_bounds__(TB, 2) k_transport(TArgs A) {
    extern __shared__ __align__(16) unsigned char smem[];
    float* T = reinterpret_cast<float*>(smem);
    float4* stg_rad = reinterpret_cast<float4*>(smem + S_TOTAL_PAD * 4);
    unsigned long long* stg_key = reinterpret_cast<unsigned long long*>(stg_rad + STG);
    Slots* SL = reinterpret_cast<Slots*>(stg_key + STG);
    StepRec* SR = reinterpret_cast<StepRec*>(SL + 1);
    StashRec* stash = reinterpret_cast<StashRec*>(SR + 1);
    uint16_t (*lists)[TB] = reinterpret_cast<uint16_t (*)[TB]>(stash + STASH);
    // What decides a barrier is read by every thread at the top of an iteration and
    // written only where a barrier lies on either side: s_want, s_hungry and s_done
    // below, s_free and s_ln by turns (par).
    __shared__ int s_sn, s_stn, s_nprim, s_done, s_hungry, s_want;
    __shared__ uint32_t s_ln[2][NLIST], s_free[2][TW], cnt[24], s_got[4];
    __shared__ unsigned long long s_flush, s_spill;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const unsigned lt = (1u << lane) - 1u;
    for (int i = tid; i < S_TOTAL; i += TB) T[i] = A.tab.small[i];
    if (tid < 24) cnt[tid] = 0;
    if (tid < 2 * NLIST) s_ln[tid / NLIST][tid % NLIST] = 0;
    if (tid < TW) s_free[0][tid] = 32u;
    if (tid == 0) { s_sn = 0; s_stn = 0; s_nprim = 0; s_done = 0; s_hungry = 0; s_want = 1; }
    DevState* S = A.st;
    Blk b{T, SL, SR, stg_rad, stg_key, &s_sn, cnt, stash, &s_stn, lists, nullptr};
    // primaries a block holds at a time: its share, at most half its slots
    const int quota = (int)min((uint32_t)TB / 2, (A.np + gridDim.x - 1) / gridDim.x);
    Dep dep{0.0, 0u};
    unsigned long long nsteps = 0;
    bool active = false, busy = false, idle = false, left = true;    // all but active: thread 0
    uint32_t par = 0;
    unsigned sleep_ns = 64;
    unsigned long long idle_since = 0;
    __syncthreads();

    for (uint32_t it = 0;; ++it) {
        // 0) here all of the last iteration is done: staging, stash and free slots
        //    are at rest until the interaction phase
        int rn = s_sn, stn = min(s_stn, STASH);
        if (rn >= STG_FLUSH || s_done) {
            if (tid == 0) s_flush = atomicAdd(&S->rad_next.v, (unsigned long long)rn);
            __syncthreads();
            if (tid == 0) s_sn = 0;                              // all have read it
            const unsigned long long base = s_flush;
            int ndrop = 0;
            for (int i = tid; i < rn; i += TB) {
                const unsigned long long slot = base + (unsigned long long)i;
                if (slot < A.max_rad) { A.rad[slot] = stg_rad[i]; A.key[slot] = stg_key[i]; }
                else ndrop++;
            }
            if (ndrop) atomicAdd(&S->rad_drop, (unsigned long long)ndrop);
            if (s_done) break;
        }
        // refill: 1) the stash (LIFO)
        int nfree = 0, rank = 0;
#pragma unroll
        for (int k = 0; k < TW; ++k) { const int f = (int)s_free[par][k]; if (k < w) rank += f; nfree += f; }
        rank += __popc(__ballot_sync(0xffffffffu, !active) & lt);
        const int share = s_hungry && TB - nfree >= SHARE ? min(SHARE, stn) : 0;
        const int take = min(nfree, stn - share);
        if (!active && rank < take) { load_secondary(*SL, tid, stash[stn - 1 - rank]); active = true; }
        stn -= take;
        // to the queue: a share for idle blocks, or a stash above its level
        int n_out = share;
        if (A.stash_spill && stn >= TW / 2 * (int)A.stash_spill) n_out = max(n_out, stn - TW / 2 * (int)A.stash_keep);
        if (n_out > 0) {
            if (tid == 0) s_spill = atomicAdd(&S->sec_qtail.v, (uint32_t)n_out);
            __syncthreads();
            for (int k = tid; k < n_out; k += TB) push_global(A, s_spill + k, stash[stn - n_out + k]);
            stn -= n_out;
        }
        int nact = TB - nfree + take;
        // 2) the global queue and 3) new primaries
        const bool poll = nact == 0 || (it & A.poll_mask) == 0u;
        const bool want = s_want != 0;
        if (nfree > take && (poll || want)) {
            if (tid == 0) {
                uint32_t base = 0, got = 0, pb = 0, pg = 0;
                const uint32_t k = (uint32_t)(nfree - take);
                if (poll) {
                    uint32_t lim = min(*(volatile uint32_t*)&S->sec_qtail.v, A.max_sec);
                    uint32_t h = *(volatile uint32_t*)&S->sec_head.v;
                    while (h < lim) {
                        uint32_t n = min(min(k, lim - h), (uint32_t)QTAKE);
                        uint32_t old = atomicCAS(&S->sec_head.v, h, h + n);
                        if (old == h) { base = h; got = n; break; }
                        h = old;
                    }
                }
                if (want && k > got) {
                    const uint32_t n = min(min(k - got, A.prim_take * TW), (uint32_t)(quota - s_nprim));
                    const uint32_t old = atomicAdd(&S->prim_next.v, n);
                    if (old < A.np) { pg = min(n, A.np - old); pb = old; }
                    if (old + n >= A.np) left = false;
                    s_nprim += (int)pg;                          // read by this thread alone until phase C
                }
                s_got[0] = base; s_got[1] = got; s_got[2] = pb; s_got[3] = pg;
            }
            __syncthreads();
            const int got = (int)s_got[1], pg = (int)s_got[3], r2 = rank - take;
            if (!active && r2 >= 0 && r2 < got) {
                const SecRec* rec = A.secq + s_got[0] + r2;
                unsigned long long t0 = gtime();
                bool ok = true;
                // bounded wait for the record's publication; once one wait has
                // run out the run is failed and no lane waits again
                while (*(volatile const uint32_t*)&rec->meta.z != A.epoch) {
                    if ((*(volatile uint32_t*)&S->err & DERR_QUEUE_WAIT) || gtime() - t0 > A.ready_ns) {
                        atomicOr(&S->err, DERR_QUEUE_WAIT);
                        ok = false;
                        break;
                    }
                    __nanosleep(64);
                }
                __threadfence();
                if (ok) {
                    float4 pe = __ldcg(&rec->pe);
                    float4 dr = __ldcg(&rec->dir);
                    uint4 mt = __ldcg(&rec->meta);
                    load_secondary(*SL, tid, StashRec{pe.x, pe.y, pe.z, pe.w, dr.x, dr.y, dr.z, mt.x, mt.y});
                    active = true;
                }
            } else if (!active && r2 >= got && r2 < got + pg) {
                start_primary(A, *SL, tid, s_got[2] + (uint32_t)(r2 - got));
                active = true;
            }
            nact += got + pg;                                    // (records that never came count until the next refill)
        }
        if (nact == 0) {
            // nothing to do and an empty stash: idle
            if (tid == 0) {
                if (busy) { busy = false; atomicSub(&S->busy.v, 1u); idle_since = gtime(); }
                if (!idle) { idle = true; atomicAdd(&S->idle.v, 1u); }
                uint32_t lim = min(*(volatile uint32_t*)&S->sec_qtail.v, A.max_sec);
                bool done = *(volatile uint32_t*)&S->prim_next.v >= A.np && *(volatile uint32_t*)&S->sec_head.v >= lim &&
                            *(volatile uint32_t*)&S->busy.v == 0u;
                if (idle_since == 0) idle_since = gtime();
                if (!done && gtime() - idle_since > A.idle_ns) { atomicOr(&S->err, DERR_IDLE_WAIT); done = true; }
                if (done) { s_done = 1; atomicSub(&S->idle.v, 1u); }
                else { __nanosleep(sleep_ns); sleep_ns = min(sleep_ns * 2, 8192u); }
                s_stn = 0;
                s_want = left && s_nprim < quota;
            }
            __syncthreads();
            continue;
        }
        if (tid == 0) {
            if (!busy) { busy = true; atomicAdd(&S->busy.v, 1u); }
            if (idle) { idle = false; atomicSub(&S->idle.v, 1u); }
            sleep_ns = 64;
            idle_since = 0;
        }
        // A) move
        b.ln = s_ln[par];
        {
            int k = -1;
            const bool was = active;
            if (nact > NREC / 4) {
                if (active) k = move(A, b, tid, dep, nsteps, active, stn > 0 ? MOVE_STEPS : MOVE_STEPS_FEW);
            } else {
                // Few electrons, most warps idle: the draws of a run do not depend on the flight,
                // so all threads draw the next 4, 8 or 16 steps of every electron side by
                // side, and the electron's own thread is left with the rotations.
                XS x;
                const int go = active ? begin_move(A, b, tid, dep, x) : 1;
                if (go) active = false;
                if (go == 2) k = L_SPUR;
                if (go == 0) {
                    SL->xi[tid] = x.xi; SL->xic[tid] = x.xic; SL->xicv[tid] = x.xicv; SL->xicvd[tid] = x.xicvd;
                    SL->stot[tid] = x.s_tot; SL->lam[tid] = x.lambda; SL->fE[tid] = x.fE; SL->iE[tid] = x.iE;
                }
                __syncwarp();
                const int at = push_list(b, L_MOVE, go == 0, (uint32_t)tid, lane);
                __syncthreads();
                const int na = (int)b.ln[L_MOVE], lg = na <= NREC / 16 ? 4 : na <= NREC / 8 ? 3 : 2;
                for (int t = tid; t < na << lg; t += TB) {
                    const int s = b.list[L_MOVE][t >> lg];
                    const uint32_t nd = SL->nd[s];
                    const float4 u = draw4_nc(nd + 4u * (uint32_t)(t & ((1 << lg) - 1)), SL->sub[s], SL->pid[s], A.k0, A.k1);
                    const Step r = draw_step(T, u, SL->lam[s], SL->iE[s], SL->fE[s], SL->stot[s], SL->xi[s], SL->xic[s],
                                             SL->xicv[s], SL->xicvd[s]);
                    SR->dist[t] = r.dist; SR->ce[t] = r.ce; SR->se[t] = r.se; SR->sp[t] = r.sp; SR->cp[t] = r.cp;
                    SR->kind[t] = r.kind;
                }
                __syncthreads();
                if (go == 0) {
                    Flight f;
                    f.load(*SL, tid, A);
                    bool esc = false;
                    for (int t = at << lg; t < (at + 1) << lg; ++t) {
                        const Step r{SR->dist[t], SR->ce[t], SR->se[t], SR->sp[t], SR->cp[t], SR->kind[t]};
                        if (f.step(r, A.box, k, esc)) break;
                    }
                    k = end_move(A, b, tid, dep, nsteps, f, x.t, x.meta, k, esc, active);
                }
            }
            __syncwarp();
#pragma unroll
            for (int q = 0; q < 3; ++q) push_list(b, q, k == q, (uint32_t)tid, lane);
            push_list(b, L_SPUR, k == L_SPUR, (uint32_t)tid | (SPUR_THERM << 8), lane);
            const unsigned ended = __ballot_sync(0xffffffffu, was && !active && SL->sub[tid] == 0u);
            const unsigned fm = __ballot_sync(0xffffffffu, !active);
            if (lane == 0) {
                s_free[par ^ 1u][w] = (uint32_t)__popc(fm);
                if (ended) atomicSub(&s_nprim, __popc(ended));
            }
        }
        __syncthreads();
        if (tid == 0) s_stn = stn;
        if (tid < NLIST) s_ln[par ^ 1u][tid] = 0;                // the next iteration's
        // B) interactions: chunks of 32 of one kind
        {
            const int n0 = (int)(b.ln[L_ION] + 31u) / 32, n1 = n0 + (int)(b.ln[L_EXC] + 31u) / 32;
            const int n2 = n1 + (int)(b.ln[L_VIB] + 31u) / 32;
            for (int c = w; c < n2; c += TW) {
                const int kind = c < n0 ? L_ION : c < n1 ? L_EXC : L_VIB;
                const uint32_t at = (uint32_t)(c - (kind == L_ION ? 0 : kind == L_EXC ? n0 : n1)) * 32u + lane;
                const bool on = at < b.ln[kind];
                const int s = on ? b.list[kind][at] : 0;
                int sp = SPUR_NONE;
                if (kind == L_VIB) { if (on) vibrate(A, b, s, dep); continue; }
                if (on) sp = kind == L_ION ? ionise(A, b, s, dep) : excite(A, b, s, dep);
                __syncwarp();
                push_list(b, L_TRACKED, sp == SPUR_TRACKED, (uint32_t)s, lane);
                push_list(b, L_SPUR, sp == SPUR_LOCAL || sp == SPUR_AUTO, (uint32_t)s | ((uint32_t)sp << 8), lane);
            }
        }
        __syncthreads();
        // C) spurs, the tracked ones with their secondary
        if (tid == TB - 1) s_hungry = *(volatile uint32_t*)&S->idle.v != 0u;
        if (tid == 0) s_want = left && s_nprim < quota;
        {
            const uint32_t nt = b.ln[L_TRACKED], ns = b.ln[L_SPUR];
            const int n0 = (int)(nt + 31u) / 32, n1 = n0 + (int)(ns + 31u) / 32;
            for (int c = w; c < n1; c += TW) {
                if (c < n0) {
                    const uint32_t at = (uint32_t)c * 32u + lane;
                    const bool on = at < nt;
                    const unsigned m = __ballot_sync(0xffffffffu, on);
                    // every emission takes a sec_buf index (counters[6]); asked for
                    // before the spur, which hides the round trip
                    uint32_t base = 0;
                    if (lane == 0) base = atomicAdd(&S->sec_tail.v, (uint32_t)__popc(m));
                    base = __shfl_sync(0xffffffffu, base, 0);
                    if (on) spur_tracked(A, b, b.list[L_TRACKED][at], base + __popc(m & lt));
                } else {
                    const uint32_t at = (uint32_t)(c - n0) * 32u + lane;
                    if (at < ns) { const uint32_t v = b.list[L_SPUR][at]; spur(A, b, (int)(v & 255u), (int)(v >> 8)); }
                }
            }
        }
        par ^= 1u;
        __syncthreads();
    }
    for (int o = 16; o; o >>= 1) {
        dep.e += __shfl_xor_sync(0xffffffffu, dep.e, o);
        dep.n += __shfl_xor_sync(0xffffffffu, dep.n, o);
        nsteps += __shfl_xor_sync(0xffffffffu, nsteps, o);
    }
    if (lane == 0) {
        atomicAdd(&S->dep_f64, dep.e);
        atomicAdd(&S->steps, nsteps);
        atomicAdd(&cnt[D_DOSE], dep.n);
    }
    __syncthreads();
    if (tid < 24 && cnt[tid]) {
        uint32_t v = cnt[tid];
        if (tid < 8) atomicAdd(&S->counters[tid], v);
        else if (tid < 16) atomicAdd(&S->sec_stats[tid - 8], v);
        else atomicAdd(&S->dbg[tid - 16], v);
    }
}

// ---------------------------------------------------------------- canonical order
// Histogram of stored entries per primary.
__global__ void k_pid_hist(const unsigned long long* key, unsigned long long n, uint32_t* cnt) {
    unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x;
    unsigned long long stride = (unsigned long long)gridDim.x * blockDim.x;
    for (; i < n; i += stride) atomicAdd(&cnt[(uint32_t)(key[i] >> 34)], 1u);
}

// Exclusive scan of n counts (+ add each) into off[0..n], one block: 4096 at a time,
// four consecutive ones per thread (9 us for 65,536; with a run of counts per thread and
// one thread adding the runs up, 128 us).
template <class T>
__device__ __forceinline__ void scan_block(const uint32_t* cnt, uint32_t n, uint32_t add, T* off) {
    __shared__ unsigned long long wsum[32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    unsigned long long carry = 0;
    for (uint32_t base = 0; base < n; base += 4096) {
        const uint32_t i = base + 4 * threadIdx.x;
        unsigned long long v[4], sum = 0;
#pragma unroll
        for (int k = 0; k < 4; ++k) { v[k] = i + k < n ? (unsigned long long)cnt[i + k] + add : 0ull; sum += v[k]; }
        unsigned long long x = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) { const unsigned long long u = __shfl_up_sync(0xffffffffu, x, o); if (lane >= o) x += u; }
        __syncthreads();
        if (lane == 31) wsum[w] = x;
        __syncthreads();
        unsigned long long before = carry + x - sum;
        for (int q = 0; q < 32; ++q) { if (q < w) before += wsum[q]; carry += wsum[q]; }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if (i + k < n) off[i + k] = (T)before;
            before += v[k];
        }
    }
    if (threadIdx.x == 0) off[n] = (T)carry;
}
__global__ void __launch_bounds__(1024) k_scan(const uint32_t* cnt, uint32_t n, unsigned long long* off) {
    scan_block(cnt, n, 0u, off);
}

// ---- canonical order without a sort.  A particle numbers its entries from 0, so an
// entry's place is the number of entries of the particles before its own plus
// its number: count per (primary, secondary), scan, scatter.  Needs every entry
// stored; a run that dropped some sorts (launch_canon).
// Measured on 5.3 M entries of 4096 x 10 keV: 910 us by per-primary bitonic
// sorts (691 of them the sorts), 140 us now; 65,536 mixed: 7.1 -> 1.4 ms.

// first particle of each primary: scan of (secondaries + 1)
__global__ void __launch_bounds__(1024) k_particles(const uint32_t* nsec, uint32_t np, uint32_t* first) {
    scan_block(nsec, np, 1u, first);
}

__device__ __forceinline__ unsigned long long stored_of(const CanonArgs& c) {
    const unsigned long long n = c.st->rad_next.v;
    return n < c.max_rad ? n : c.max_rad;
}
__device__ __forceinline__ uint32_t particle_of(const CanonArgs& c, unsigned long long key) {
    return c.first[(uint32_t)(key >> 34)] + ((uint32_t)(key >> 17) & 0x1ffffu);
}

__global__ void k_count(CanonArgs c) {
    const unsigned long long n = stored_of(c);
    for (unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; i < n;
         i += (unsigned long long)gridDim.x * blockDim.x) {
        const uint32_t q = particle_of(c, c.key[i]);
        if (q < c.cap) atomicAdd(&c.cnt[q], 1u);
    }
}

// sums of CB equal shares of the counts, then the scan of each share from the sums before it
constexpr int CBLK = 592, CTHR = 256;
__global__ void __launch_bounds__(CTHR) k_share_sum(CanonArgs c) {
    __shared__ uint32_t s[CTHR / 32];
    const uint32_t m = min(c.first[c.np], c.cap), per = (m + CBLK - 1) / CBLK;
    const uint32_t lo = min(blockIdx.x * per, m), hi = min(lo + per, m);
    uint32_t v = 0;
    for (uint32_t i = lo + threadIdx.x; i < hi; i += CTHR) v += c.cnt[i];
    for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t t = 0;
        for (int k = 0; k < CTHR / 32; ++k) t += s[k];
        c.share[blockIdx.x] = t;
    }
}
__global__ void __launch_bounds__(CTHR) k_share_scan(CanonArgs c) {
    __shared__ uint32_t s[CTHR / 32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const uint32_t m = min(c.first[c.np], c.cap), per = (m + CBLK - 1) / CBLK;
    const uint32_t lo = min(blockIdx.x * per, m), hi = min(lo + per, m);
    uint32_t before = 0;
    for (uint32_t k = threadIdx.x; k < blockIdx.x; k += CTHR) before += c.share[k];
    for (int o = 16; o; o >>= 1) before += __shfl_xor_sync(0xffffffffu, before, o);
    if (lane == 0) s[w] = before;
    __syncthreads();
    before = 0;
    for (int k = 0; k < CTHR / 32; ++k) before += s[k];
    for (uint32_t b = lo; b < hi; b += CTHR) {
        const uint32_t i = b + threadIdx.x, own = i < hi ? c.cnt[i] : 0u;
        uint32_t x = own;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) { const uint32_t u = __shfl_up_sync(0xffffffffu, x, o); if (lane >= o) x += u; }
        __syncthreads();
        if (lane == 31) s[w] = x;
        __syncthreads();
        uint32_t at = before + x - own;
        for (int k = 0; k < CTHR / 32; ++k) { if (k < w) at += s[k]; before += s[k]; }
        if (i < hi) c.cnt[i] = at;                               // in place: counts become offsets
    }
}

// Entries of a primary, at most: what the sort of launch_canon holds in shared memory.  A
// transport whose entries are placed by counting could have more, but is refused the same, so
// that a primary does not pass or fail by whether another one's entries were dropped.
constexpr int SEG_MAX = 8192;
// entries to their places; the primaries' offsets and the longest segment
__global__ void k_place(CanonArgs c) {
    const unsigned long long n = stored_of(c), stride = (unsigned long long)gridDim.x * blockDim.x;
    const unsigned long long t = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x;
    for (unsigned long long i = t; i < n; i += stride) {
        const unsigned long long key = c.key[i];
        const uint32_t q = particle_of(c, key);
        if (q >= c.cap) continue;
        const unsigned long long at = (unsigned long long)c.cnt[q] + (key & 0x1ffffull);
        if (at < n) c.out[at] = c.rad[i];
    }
    uint32_t longest = 0;
    for (unsigned long long p = t; p <= c.np; p += stride) {
        auto off = [&](uint32_t k) -> unsigned long long {
            const uint32_t q = c.first[k];
            return k == c.np || q >= c.cap ? n : c.cnt[q];
        };
        const unsigned long long a = off((uint32_t)p);
        c.off[p] = a;
        if (p < c.np) longest = max(longest, (uint32_t)(off((uint32_t)p + 1) - a));
    }
    for (int o = 16; o; o >>= 1) longest = max(longest, __shfl_xor_sync(0xffffffffu, longest, o));
    if ((threadIdx.x & 31) == 0 && longest) {
        atomicMax(&c.red[2], (unsigned long long)longest);
        if (longest > (uint32_t)SEG_MAX) atomicOr(c.err, DERR_SEG_SORT);
    }
}

// everything a transport starts from at zero, in one launch
__global__ void k_clear(ClearArgs c) {
    const size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x, stride = (size_t)gridDim.x * blockDim.x;
    uint4* d = reinterpret_cast<uint4*>(c.dose);
    for (size_t i = t; i < c.nvox / 4; i += stride) d[i] = make_uint4(0u, 0u, 0u, 0u);
    for (size_t i = c.nvox / 4 * 4 + t; i < c.nvox; i += stride) c.dose[i] = 0u;
    uint4* q = reinterpret_cast<uint4*>(c.cnt);
    for (size_t i = t; i < c.cap / 4; i += stride) q[i] = make_uint4(0u, 0u, 0u, 0u);
    for (size_t i = c.cap / 4 * 4 + t; i < c.cap; i += stride) c.cnt[i] = 0u;
    for (size_t i = t; i < c.np; i += stride) c.nsec[i] = 0u;
    uint32_t* st = reinterpret_cast<uint32_t*>(c.st);
    for (size_t i = t; i < sizeof(DevState) / 4; i += stride) st[i] = 0u;
    if (t < 4) c.red[t] = 0ull;
    if (t == 4) *c.err = 0u;
}

__global__ void k_scatter(const unsigned long long* key, unsigned long long n, const unsigned long long* off,
                          uint32_t* cur, uint32_t* perm) {
    unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x;
    unsigned long long stride = (unsigned long long)gridDim.x * blockDim.x;
    for (; i < n; i += stride) {
        uint32_t p = (uint32_t)(key[i] >> 34);
        perm[off[p] + atomicAdd(&cur[p], 1u)] = (uint32_t)i;
    }
}

// One block per primary: sort its entries by key (bitonic, shared memory) and
// write them to the canonical buffer.
__global__ void __launch_bounds__(1024) k_segsort(const unsigned long long* key, const float4* rad,
                                                  const uint32_t* perm, const unsigned long long* off,
                                                  float4* out, uint32_t* err) {
    extern __shared__ __align__(16) unsigned char seg_smem[];
    unsigned long long* sk = reinterpret_cast<unsigned long long*>(seg_smem);
    uint32_t* si = reinterpret_cast<uint32_t*>(sk + SEG_MAX);
    uint32_t p = blockIdx.x;
    unsigned long long s = off[p], e = off[p + 1];
    uint32_t len = (uint32_t)(e - s);
    if (len == 0) return;
    if (len > SEG_MAX) { if (threadIdx.x == 0) atomicOr(err, DERR_SEG_SORT); return; }
    uint32_t n2 = 1;
    while (n2 < len) n2 <<= 1;
    for (uint32_t i = threadIdx.x; i < n2; i += blockDim.x) {
        if (i < len) { uint32_t ix = perm[s + i]; sk[i] = key[ix]; si[i] = ix; }
        else { sk[i] = ~0ull; si[i] = 0; }
    }
    __syncthreads();
    for (uint32_t k = 2; k <= n2; k <<= 1) {
        for (uint32_t j = k >> 1; j > 0; j >>= 1) {
            for (uint32_t i = threadIdx.x; i < n2; i += blockDim.x) {
                uint32_t l = i ^ j;
                if (l > i) {
                    bool up = (i & k) == 0;
                    unsigned long long a = sk[i], c = sk[l];
                    if ((a > c) == up) { sk[i] = c; sk[l] = a; uint32_t t = si[i]; si[i] = si[l]; si[l] = t; }
                }
            }
            __syncthreads();
        }
    }
    for (uint32_t i = threadIdx.x; i < len; i += blockDim.x) out[s + i] = rad[si[i]];
}

// n_therm (non-escaped primaries) and the dose-grid sum
__global__ void k_reduce(const float* results, uint32_t np, const uint32_t* dose, uint32_t nvox,
                         unsigned long long* out) {
    unsigned long long sd = 0;
    uint32_t nt = 0;
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x, stride = gridDim.x * blockDim.x;
    const uint4* d4 = reinterpret_cast<const uint4*>(dose);
    for (uint32_t v = i; v < nvox / 4; v += stride) {
        const uint4 q = d4[v];
        sd += (unsigned long long)q.x + q.y + q.z + q.w;
    }
    for (uint32_t v = nvox / 4 * 4 + i; v < nvox; v += stride) sd += dose[v];
    for (uint32_t v = i; v < np; v += stride) nt += (__float_as_uint(results[8ull * v + 5]) == 0u);
    for (int o = 16; o; o >>= 1) {
        sd += __shfl_xor_sync(0xffffffffu, sd, o);
        nt += __shfl_xor_sync(0xffffffffu, nt, o);
    }
    if ((threadIdx.x & 31) == 0) { atomicAdd(&out[0], sd); atomicAdd(&out[1], (unsigned long long)nt); }
}

// ------------------------------------------------------------------ host side
size_t transport_smem_bytes() {
    return S_TOTAL_PAD * 4 + STG * 24 + sizeof(Slots) + sizeof(StepRec) + STASH * sizeof(StashRec) + NLIST * TB * 2;
}

// resident CTAs of k_transport on `device` (the current device); the shared
// memory attribute is set on each device the first time
int transport_blocks(int device, uint32_t ctas_per_sm) {
    static DeviceOnce attr;
    attr.run([] {
        // all of the SM's memory as shared memory: with the split the previous
        // kernel left, a second CTA may not fit beside the first
        cudaError_t e = cudaFuncSetAttribute(k_transport, cudaFuncAttributePreferredSharedMemoryCarveout,
                                             cudaSharedmemCarveoutMaxShared);
        if (e != cudaSuccess) return e;
        return cudaFuncSetAttribute(k_transport, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)transport_smem_bytes());
    });
    int sms = 0, per = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_transport, TB, transport_smem_bytes());
    if (per < 1) per = 1;
    if (ctas_per_sm && (int)ctas_per_sm < per) per = (int)ctas_per_sm;
    return sms * per;
}

cudaError_t launch_transport(const TArgs& a, int blocks, cudaStream_t s) {
    k_transport<<<blocks, TB, transport_smem_bytes(), s>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_canon(const unsigned long long* key, const float4* rad, unsigned long long n, uint32_t np,
                         uint32_t* cnt, unsigned long long* off, uint32_t* cur, uint32_t* perm, float4* out,
                         uint32_t* err, cudaStream_t s) {
    cudaError_t e = cudaMemsetAsync(cnt, 0, (size_t)np * 4, s);
    if (e == cudaSuccess) e = cudaMemsetAsync(cur, 0, (size_t)np * 4, s);
    if (e != cudaSuccess) return e;
    if (n) k_pid_hist<<<1184, 256, 0, s>>>(key, n, cnt);
    k_scan<<<1, 1024, 0, s>>>(cnt, np, off);
    if (n) {
        k_scatter<<<1184, 256, 0, s>>>(key, n, off, cur, perm);
        static DeviceOnce attr;
        e = attr.run([] {
            return cudaFuncSetAttribute(k_segsort, cudaFuncAttributeMaxDynamicSharedMemorySize, SEG_MAX * 12);
        });
        if (e != cudaSuccess) return e;
        k_segsort<<<np, 1024, SEG_MAX * 12, s>>>(key, rad, perm, off, out, err);
    }
    return cudaGetLastError();
}

cudaError_t launch_scan_u32(const uint32_t* cnt, uint32_t n, unsigned long long* off, cudaStream_t s) {
    k_scan<<<1, 1024, 0, s>>>(cnt, n, off);
    return cudaGetLastError();
}

cudaError_t launch_reduce(const float* results, uint32_t np, const uint32_t* dose, uint32_t nvox,
                          unsigned long long* out, cudaStream_t s) {
    k_reduce<<<592, 256, 0, s>>>(results, np, dose, nvox, out);
    return cudaGetLastError();
}

cudaError_t launch_clear(const ClearArgs& c, cudaStream_t s) {
    k_clear<<<592, 256, 0, s>>>(c);
    return cudaGetLastError();
}

cudaError_t launch_place(const CanonArgs& c, cudaStream_t s) {
    k_particles<<<1, 1024, 0, s>>>(c.nsec, c.np, c.first);
    k_count<<<1184, 256, 0, s>>>(c);
    k_share_sum<<<CBLK, CTHR, 0, s>>>(c);
    k_share_scan<<<CBLK, CTHR, 0, s>>>(c);
    k_place<<<1184, 256, 0, s>>>(c);
    return cudaGetLastError();
}

}  // namespace wg
