// irt.cu -- Karamitros 2011 9-reaction IRT radiolysis chemistry to 1 us.
//
// Follows public/irt-worker.js of allaunthefox/webgpu-dna (species and
// reaction tables :191-286, sampleIRT :116-184 with SamplePDC :91-113, erfcinv
// :31-39, erfcx :53-88, the per-primary event loop :470-667 and pairWithAlive
// :430-465).  The reference runs the primaries one after another on one CPU
// thread; here a warp, or several where there are few tracks, owns one track (primary)
// at a time and the warps of a persistent grid pull tracks from a counter:
//
// * load: entries of the track (codes 4/7 skipped, 7 counted as initial H2)
//   are displaced in f64 with the thermalisation Gaussians, 32 at a time;
// * initial pairing: tiles of 32 particles held in lane registers, the partner
//   j broadcast to all lanes; one Philox block gives the acceptance draws of
//   four consecutive partners;
// * sort: the initial events of a track in (t, i, j) order, one block per
//   track, in shared memory;
// * events: the sorted initial events merged with a heap of product events
//   ordered by (t, i, j); the product re-pairing (pairWithAlive) is spread over
//   the lanes of the track's warps.
//
// Random draws are keyed by what they are for (track, particle, pair), so the
// result does not depend on scheduling; the CPU oracle uses the same streams:
//   load of particle k            philox(blk, k, pid, 2), 53-bit doubles
//   acceptance of pair i<j         philox(j>>2, i, pid, 3), word j&3
//   SamplePDC trial t of (i, j)    philox(i, j, pid, 4 | t<<4)
//   product idx, partner jj        philox(idx, jj, pid, 5): Box-Muller radii
//                                  x,y,z + acceptance; philox(.., 5 | 1<<4):
//                                  Box-Muller angles.
#include <cstring>

#include <algorithm>

#include "irt.cuh"
#include "dmath.cuh"

namespace wg {


__constant__ IrtConst c_irt;


constexpr uint32_t FULL = 0xffffffffu;
constexpr int IB = 128;                  // threads per block (4 warps)

__device__ __forceinline__ double erfcinv_(double x) {                       // :31-39
    if (x <= 0 || x >= 2) return 0;
    double p = x > 1 ? 2 - x : x;
    double t = sqrt(-2 * log_(p / 2));
    double y = t - (2.515517 + 0.802853 * t + 0.010328 * t * t) /
                   (1 + 1.432788 * t + 0.189269 * t * t + 0.001308 * t * t * t);
    y *= 0.7071067811865475;
    return x > 1 ? -y : y;
}

__constant__ double c_erfcx[28] = {
    -1.3026537197817094, 6.4196979235649026e-1, 1.9476473204185836e-2, -9.561514786808631e-3,
    -9.46595344482036e-4, 3.66839497852761e-4, 4.2523324806907e-5, -2.0278578112534e-5,
    -1.624290004647e-6, 1.303655835580e-6, 1.5626441722e-8, -8.5238095915e-8,
    6.529054439e-9, 5.059343495e-9, -9.91364156e-10, -2.27365122e-10,
    9.6467911e-11, 2.394038e-12, -6.886027e-12, 8.94487e-13,
    3.13092e-13, -1.12708e-13, 3.81e-16, 7.106e-15,
    -1.523e-15, -9.4e-17, 1.21e-16, -2.8e-17};

// (out of line and rolled: the undecided trials that need it are rare, and the kernels'
// instructions have to stay in the SM's cache)
__device__ __noinline__ double erfcx_pos(double x) {                                      // :53-88, x >= 0
    if (x >= 6) {
        double f = 0;
#pragma unroll 1
        for (int n = 30; n >= 1; --n) f = (0.5 * n) / (x + f);
        return 0.5641895835477563 / (x + f);
    }
    double t = 2.0 / (2.0 + x);
    double ty = 4 * t - 2;
    double d = 0, dd = 0;
#pragma unroll 1
    for (int j = 27; j > 0; --j) { double tmp = d; d = ty * d - dd + c_erfcx[j]; dd = tmp; }
    return t * exp_(0.5 * (c_erfcx[0] + ty * d) - dd);
}
__device__ __forceinline__ double erfcx_(double x) {
    if (x < 0) return 2 * exp_(x * x) - erfcx_pos(-x);
    return erfcx_pos(x);
}

// f32 erfcx for z >= 0, used only to bound the f64 value: the reference's
// Chebyshev form (first 14 coefficients) below 6, the asymptotic series
// (1 / (z sqrt(pi))) sum (-1)^k (2k-1)!! / (2 z^2)^k to k = 7 above.  Its
// largest relative error against the f64 form is 3.3e-7 (z on a 1e-5 grid
// to 200 and log-spaced to 1e8, with a 1-ulp expf).
__constant__ float c_erfcx_f[14] = {
    -1.3026537197817094f, 6.4196979235649026e-1f, 1.9476473204185836e-2f, -9.561514786808631e-3f,
    -9.46595344482036e-4f, 3.66839497852761e-4f, 4.2523324806907e-5f, -2.0278578112534e-5f,
    -1.624290004647e-6f, 1.303655835580e-6f, 1.5626441722e-8f, -8.5238095915e-8f,
    6.529054439e-9f, 5.059343495e-9f};

__device__ __forceinline__ float erfcx_f(float z) {
    if (z >= 6.0f) {
        float iz = __frcp_rn(z);
        float h = 0.5f * iz * iz;
        float s = 1.0f - 13.0f * h;
        s = 1.0f - 11.0f * h * s; s = 1.0f - 9.0f * h * s; s = 1.0f - 7.0f * h * s;
        s = 1.0f - 5.0f * h * s; s = 1.0f - 3.0f * h * s; s = 1.0f - h * s;
        return s * 0.5641895835f * iz;
    }
    float t = __fdividef(2.0f, 2.0f + z), ty = 4.0f * t - 2.0f, d = 0.0f, dd = 0.0f;
    for (int j = 13; j > 0; --j) { float tmp = d; d = fmaf(ty, d, c_erfcx_f[j] - dd); dd = tmp; }
    return t * __expf(0.5f * fmaf(ty, d, c_erfcx_f[0]) - dd);
}

// SamplePDC (:91-113): what a trial needs of its pair.  The f64 members give
// the winner's X and the undecided trials; the f32 ones the brackets.
struct PdcPair {
    double pq, M;                      // p + q M and M (:92-95)
    float thr, pqf, Mf, t2f, bbf, af, bf;
};
__device__ __forceinline__ PdcPair pdc_pair(double a, double b) {
    const double r = sqrt(2.0 * b / a);
    const double p = 2.0 * r, q = 2.0 / r;
    PdcPair P;
    P.M = fmax(1.0 / (a * a), 3.0 * b / a);
    P.pq = p + q * P.M;
    P.thr = (float)(p / P.pq);
    P.pqf = (float)P.pq; P.Mf = (float)P.M; P.t2f = (float)(2.0 * b / a); P.bbf = (float)(b * b);
    P.af = (float)a; P.bf = (float)b;
    return P;
}
// X of a trial (:97-103) from its first two words
__device__ __forceinline__ double pdc_x(double a, double b, double pq, double M, uint32_t wx, uint32_t wy) {
    const double U1 = u01d(wx, wy), p = 2.0 * sqrt(2.0 * b / a);
    if (U1 < p / pq) { const double h = U1 * pq / 2; return h * h; }
    const double h = 2 / ((1 - U1) * pq / M);
    return h * h;
}

// The first accepted trial of lane `src`'s pair (qi, qj), 32 trials at a time
// across the warp: in trial order, as in the sequential loop.  All 32 lanes call;
// P, a and b are read from lane src.  Returns the trial's first two words (the
// caller turns them into X), or ~0 when 10,000 trials are rejected.
//
// What bounds it: the issue slots of 60 evaluated trials per pair (42 up to the
// accepted one, 2.4 % of them accepted).  The pair's f64 square root and divisions
// are therefore done once per pair by its own lane, not by all lanes of the
// call, and a trial first meets an upper bound of lambdax that costs 30
// instructions beside its Philox block:
//   Q >= (1 - beta) (1 - h), so 1 - Q <= beta + h   (h, beta as below; any z > 0,
//   the asymptotic series of erfcx alternates), which rejects all but 2.43 %.
//   Its draws are the upper words alone (U1 and 1 - U1 within 2^-27, so X to 2.2e-4
//   and e to 2.2e-4 b^2/X relative when both exceed 1.2e-4, else the trial goes on;
//   U2 rounded down); 3 % + 1e-3 b^2/X covers that.
// Only what is left meets the bracket.  Measured in the pairing kernel (4096 x 10 keV,
// 6.5 M calls): 2.8 ms with a pair to a lane (pdc_queue), 3.7 ms by whole warps
// (pdc_find), there 5.1 ms with the bracket in every round and 6 ms with the f64
// set-up in every lane.
//
// A trial is accepted when U2 <= lambdax (X <= 2b/a) or U2 M / X <= lambdax
// (X >= 2b/a), lambdax = e (1 - Q), e = exp(-b^2/X), Q = a sqrt(pi X)
// erfcx(b/sqrt(X) + a sqrt(X)).  Each trial brackets the f64 lambdax with f32
// arithmetic (the fast reciprocal, rsqrt, divide and exp2 instructions, 2 ulp
// each; ex2 adds |x| 8.6e-8 for exp(x)):
//   U1, 1 - U1 and U2 are the 53-bit draws rounded to f32 (1.2e-7 relative, from
//   the exact integers), a draw within 1e-6 of the branch point is undecided;
//   X to 1.2e-6 relative, so b^2/X to 2e-6 and e to (4e-6 b^2/X + 2e-6);
//   z to 1e-6 relative, which moves erfcx by at most 1.2e-6 (|d ln erfcx/dz|
//   <= 1.13 and <= 1/z); with the 3.3e-7 of erfcx_f (8e-7 with the fast
//   exp) the prefactor Q is known to 4e-6, taken as 2e-5, 1 - Q to that
//   plus 1e-6;
//   for z >= 6 and b >= 0, where 1 - Q cancels, 1 - Q itself: with
//   beta = (b/sqrt(X))/z, Q = (1 - beta) S and erfcx(z) = S/(z sqrt(pi)),
//   S = 1 - h s (h = 1/(2z^2), s the asymptotic series of erfcx_f), so
//   1 - Q = beta + (1 - beta) h s, a sum of two non-negative terms known to
//   1.7e-6 and 4.2e-6 relative (1/z correctly rounded; the f32 series
//   within 2.2e-7 of h s); taken as 2e-5.  The f64 1 - Q it must bound
//   carries the rounding of Q near 1 (about 7 ulp, the continued fraction
//   of erfcx_pos within 2.2e-16), so 1e-14 is added on both sides;
// and decides when U2 (or U2 M against lambdax X) lies outside the bracket,
// itself widened by 2e-6 relative and 1e-30, with a further margin of 1e-6
// (5e-6).  Trials inside the bracket, near X = 2b/a, z < 0, or with a zero draw
// are evaluated exactly in f64.
__device__ __forceinline__ float rcp_fast(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float exp_fast(float x) {                 // 0 below 2^-126
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x * 1.4426950f));
    return r;
}

// the upper bound: false when the trial is surely rejected
__device__ __forceinline__ bool pdc_maybe(const u4& w, float thr, float hpq, float qpq, float Mf, float t2f, float af, float bf) {
    const float u = __uint2float_rd(w.x) * 0x1p-32f, v = 1.0f - u;
    const bool ca = u < thr;
    const float q = ca ? u * hpq : v * qpq;             // sqrt(X), or its reciprocal
    const float r = rcp_fast(q);
    const float hx = ca ? q : r, rs = ca ? r : q;
    const float y = bf * rs, arg = y * y, iz = rcp_fast(fmaf(af, hx, y));
    const float lam = fmaxf(exp_fast(-arg), 1e-30f) * iz * fmaf(0.5f, iz, y) * fmaf(1e-3f, arg, 1.03f);
    const float mult = hx * hx < t2f * 1.001f ? 1.0f : Mf * rs * rs;
    const bool rej = __uint2float_rd(w.z) * 0x1p-32f * mult > lam;
    return !(rej && fminf(u, v) > 1.2e-4f && bf >= 0.0f);
}
// the bracket: 0 rejected, 1 accepted, 2 undecided
__device__ __forceinline__ int pdc_bracket(const u4& w, float thr, float pqf, float Mf, float t2f, float bbf, float af, float bf) {
    const uint32_t ah = w.x >> 5, al = w.y >> 6;
    const float u1 = fmaf((float)ah, 0x1p-27f, (float)al * 0x1p-53f);
    const float v1 = fmaf((float)(0x7ffffffu - ah), 0x1p-27f, (float)(0x4000000u - al) * 0x1p-53f);   // 1 - U1
    const float u2 = fmaf((float)(w.z >> 5), 0x1p-27f, (float)(w.w >> 6) * 0x1p-53f);
    const float hx = u1 < thr ? u1 * pqf * 0.5f : __fdividef(2.0f * Mf, v1 * pqf);
    const float xf = hx * hx;
    const bool ca = xf < t2f * 0.99999f, cb = xf > t2f * 1.00001f;
    if (!(u2 > 0.0f && xf > 1e-30f && xf < 1.0e30f && (ca || cb) && fabsf(u1 - thr) > thr * 1e-6f)) return 2;
    const float rs = rsqrtf(xf);
    const float argf = bbf * rs * rs;
    float elo = 0.0f, ehi = 1e-30f;
    if (argf <= 80.0f) {
        const float ef = __expf(-argf), re = argf * 4e-6f + 2e-6f;
        elo = ef * (1.0f - re); ehi = ef * (1.0f + re);
    }
    const float sx = xf * rs;
    const float zf = bf * rs + af * sx;
    if (!(zf >= 0.0f)) return 2;
    float flo, fhi;
    if (zf >= 6.0f && bf >= 0.0f) {
        const float iz = __frcp_rn(zf), h = 0.5f * iz * iz;
        float s = 1.0f - 13.0f * h;
        s = 1.0f - 11.0f * h * s; s = 1.0f - 9.0f * h * s; s = 1.0f - 7.0f * h * s;
        s = 1.0f - 5.0f * h * s; s = 1.0f - 3.0f * h * s;
        const float omq = fmaf(af * sx * iz, h * s, bf * rs * iz);
        flo = omq * 0.99998f - 1e-14f; fhi = omq * 1.00002f + 1e-14f;
    } else {
        const float Q = af * 1.7724539f * sx * erfcx_f(zf);
        flo = 1.0f - Q * 1.00002f - 1e-6f; fhi = 1.0f - Q * 0.99998f + 1e-6f;
    }
    const float Llo = elo * fmaxf(flo, 0.0f) * (1.0f - 2e-6f) - 1e-30f;
    const float Lhi = ehi * fmaxf(fhi, 0.0f) * (1.0f + 2e-6f) + 1e-30f;
    if (ca) return u2 <= Llo * (1.0f - 1e-6f) ? 1 : (u2 > Lhi * (1.0f + 1e-6f) ? 0 : 2);
    const float lhs = u2 * Mf;
    return lhs <= Llo * xf * (1.0f - 5e-6f) ? 1 : (lhs > Lhi * xf * (1.0f + 5e-6f) ? 0 : 2);
}
// the trial in f64 (:97-110)
__device__ __forceinline__ bool pdc_exact(const u4& w, double da, double db) {
    const double t2 = 2.0 * db / da, r = sqrt(t2), M = fmax(1.0 / (da * da), 3.0 * db / da);
    const double pq = 2.0 * r + 2.0 / r * M;
    const double X = pdc_x(da, db, pq, M, w.x, w.y), U2 = u01d(w.z, w.w);
    // lambdax <= e: a trial that fails against e alone is rejected
    // without evaluating erfcx (same decision as the full test)
    const double e = exp_(-db * db / X);
    const double v = U2 * M / X;
    if (!((X <= t2 && U2 <= e) || (X >= t2 && v <= e))) return false;
    const double sqX = sqrt(X);
    const double lambdax = e * (1.0 - da * sqrt(3.141592653589793 * X) * erfcx_(db / sqX + da * sqX));
    return (X <= t2 && U2 <= lambdax) || (X >= t2 && v <= lambdax);
}

// One pair by the whole warp, 32 trials at a time from trial `first` on; all 32 lanes
// call.  What a pair costs this way: 59 evaluated trials (42 up to the accepted
// one), and the bracket in 54 % of the rounds, for one lane or two.
__device__ __forceinline__ uint64_t pdc_find(int src, uint32_t i, uint32_t j, uint32_t pid, const PdcPair& P, double a,
                                             double b, int lane, const uint32_t* rk, uint32_t first = 0) {
    const uint32_t qi = __shfl_sync(0xffffffffu, i, src), qj = __shfl_sync(0xffffffffu, j, src);
    const float thr = __shfl_sync(0xffffffffu, P.thr, src), pqf = __shfl_sync(0xffffffffu, P.pqf, src);
    const float Mf = __shfl_sync(0xffffffffu, P.Mf, src), t2f = __shfl_sync(0xffffffffu, P.t2f, src);
    const float bbf = __shfl_sync(0xffffffffu, P.bbf, src), af = __shfl_sync(0xffffffffu, P.af, src);
    const float bf = __shfl_sync(0xffffffffu, P.bf, src);
    const float hpq = 0.5f * pqf, qpq = __fdividef(0.5f * pqf, Mf);
#pragma unroll 1
    for (uint32_t t0 = first; t0 < 10000; t0 += 32) {
        const uint32_t trial = t0 + lane;
        const u4 w = philox_rk(qi, qj, pid, 4u | (trial << 4), rk);
        int st = trial < 10000 && pdc_maybe(w, thr, hpq, qpq, Mf, t2f, af, bf) ? 2 : 0;
        if (!__any_sync(0xffffffffu, st != 0)) continue;
        if (st != 0) st = pdc_bracket(w, thr, pqf, Mf, t2f, bbf, af, bf);
        if (__any_sync(0xffffffffu, st == 2)) {
            const double da = __shfl_sync(0xffffffffu, a, src), db = __shfl_sync(0xffffffffu, b, src);
            if (st == 2) st = pdc_exact(w, da, db) ? 1 : 0;
        }
        const unsigned m = __ballot_sync(0xffffffffu, st == 1);
        if (m) {
            const int win = __ffs(m) - 1;
            return ((uint64_t)__shfl_sync(0xffffffffu, w.x, win) << 32) | __shfl_sync(0xffffffffu, w.y, win);
        }
    }
    return ~0ull;
}

// sampleIRT (:116-184) with the acceptance draw U supplied.  Returns the
// reaction time t >= 0, -1 for no reaction, or -2 when SamplePDC must be run
// with (*pa, *pb); the caller then uses X / D for X > 0.
__device__ __forceinline__ double sample_pre(const IrtConst& C, double r0, int ri, double D, double U,
                                             double* pa, double* pb) {
    if (C.type[ri] == 0) {
        double sigma = C.sigma[ri], rc = C.rc[ri];
        if (sigma <= 0 || D <= 0) return -1;
        if (r0 <= sigma) return 0;
        double r0e = r0;
        if (rc != 0) r0e = -rc / (1 - exp_(rc / r0));
        if (r0e <= sigma) return 0;
        double Winf = sigma / r0e;
        if (U <= 0 || U >= Winf) return -1;
        double ei = erfcinv_(r0e * U / sigma);
        if (fabs(ei) < 1e-10) return -1;
        double dr = r0e - sigma;
        return 0.25 * dr * dr / (D * ei * ei);
    }
    double sigma_c = C.sigma[ri], rc = C.rc[ri];
    double b, sc_chk = sigma_c, r0_chk = r0;
    if (rc == 0) {
        b = (r0 - sigma_c) / 2;
    } else {
        double coth_r0 = 1.0 + 2.0 / expm1_(2.0 * (rc / (2 * r0)));
        b = rc / 4 * (coth_r0 - C.coth_sig[ri]);
        r0_chk = -rc / (1 - exp_(rc / r0));
        sc_chk = C.sigma_eff[ri];
    }
    if (sc_chk > r0_chk) return (C.prob[ri] > U) ? 0 : -1;
    double Winf = sc_chk / r0_chk * C.kobs[ri] / C.kdif[ri];
    if (Winf > U) { *pa = C.a_pdc[ri]; *pb = b; return -2; }
    return -1;
}

// Distance beyond which sample_pre certainly returns -1 for acceptance draw U:
//   TDC:  Winf = sigma / r0e and r0e >= r0 - max(rc,0)/2      -> r0 < sigma/U + rc/2
//   PDC:  contact needs r0 < sigma_x, Winf = sigma_x c / r0_chk with r0_chk >= r0
//         (c = kobs/kdif)                                     -> r0 < max(sigma_x, sigma_x c / U)
// with a relative and absolute safety margin for rounding.
__device__ __forceinline__ double r_acc(const IrtConst& C, int ri, double U) {
    double s = C.acc_s[ri];
    double R = fmax(s, s * C.acc_c[ri] / U) + C.acc_add[ri];
    return R * (1.0 + 1e-6) + 1e-6;
}

// Event heap on (t, packed a<<16|b): 32 children to a node, so that a warp takes a level
// in one load and a vote.  Nodes [0, HS) in shared memory, the rest in global memory.
// A binary heap of one lane took 3100 cycles per pop on a track with 2500 product events
// (9 levels, the lower ones in L2); this one 1400.
template <int HS>
struct Heap {
    double* st; uint32_t* sab; double* gt; uint32_t* gab;
    __device__ __forceinline__ double t(uint32_t k) const { return k < HS ? st[k] : gt[k - HS]; }
    __device__ __forceinline__ uint32_t ab(uint32_t k) const { return k < HS ? sab[k] : gab[k - HS]; }
    __device__ __forceinline__ void set(uint32_t k, double tv, uint32_t abv) const {
        if (k < HS) { st[k] = tv; sab[k] = abv; } else { gt[k - HS] = tv; gab[k - HS] = abv; }
    }
};
__device__ __forceinline__ bool ev_less(double t1, uint32_t x, double t2, uint32_t y) {
    return t1 != t2 ? t1 < t2 : x < y;
}
// node c, the last one, moves up to its place
template <int HS>
__device__ __forceinline__ void heap_up(const Heap<HS>& H, uint32_t c) {
    if (c == 0) return;
    const double t = H.t(c);
    const uint32_t ab = H.ab(c);
#pragma unroll 1
    while (c > 0) {
        const uint32_t p = (c - 1) >> 5;
        const double tp = H.t(p);
        const uint32_t ap = H.ab(p);
        if (!ev_less(t, ab, tp, ap)) break;
        H.set(c, tp, ap);
        c = p;
    }
    H.set(c, t, ab);
}
// by the whole warp; times are not negative, so their bit patterns are in order
template <int HS>
__device__ __forceinline__ void heap_pop(const Heap<HS>& H, uint32_t& n, int lane) {
    n--;
    if (n == 0) return;
    const double tp = H.t(n);
    const uint32_t ap = H.ab(n);
    uint32_t p = 0;
#pragma unroll 1
    for (;;) {
        const uint32_t c = 32 * p + 1 + lane;
        if (32 * p + 1 >= n) break;
        const bool in = c < n;
        const double tc = in ? H.t(c) : 0.0;
        const uint32_t ac = in ? H.ab(c) : 0u;
        const uint32_t hi = in ? (uint32_t)__double2hiint(tc) : 0xffffffffu, lo = (uint32_t)__double2loint(tc);
        unsigned m = __ballot_sync(FULL, hi == __reduce_min_sync(FULL, hi));
        if (m & (m - 1)) {                               // equal upper words: the lower ones, then a and b
            const bool s1 = m >> lane & 1;
            const uint32_t l1 = __reduce_min_sync(FULL, s1 ? lo : 0xffffffffu);
            const bool s2 = s1 && lo == l1;
            const uint32_t a1 = __reduce_min_sync(FULL, s2 ? ac : 0xffffffffu);
            m = __ballot_sync(FULL, s2 && ac == a1);
        }
        const int w = __ffs(m) - 1;
        const double tm = __shfl_sync(FULL, tc, w);
        const uint32_t am = __shfl_sync(FULL, ac, w);
        if (!ev_less(tm, am, tp, ap)) break;
        if (lane == 0) H.set(p, tm, am);
        p = 32 * p + 1 + w;
    }
    if (lane == 0) H.set(p, tp, ap);
    __syncwarp();
}

// checkpoint times of the reference timeline (:566-580), ns
__constant__ double c_cp[7] = {0.001, 0.01, 0.1, 1, 10, 100, 1000};

// Per-track storage (one track = one primary): particle slots at
// tbase(p) = 2*seg_off[p] + 64*p with capacity 2*len + 64 (len = the track's
// rad_buf entries; a track that outgrows it before the reference's CAP sets
// DERR_TRACK_SIZE), initial-event slots at ebase(p) = 16*seg_off[p] + 2048*p:
// up to ecap(p) = 8*len + 1024 events (DERR_HEAP beyond), twice that room for
// the power-of-two padding of the sort.
__device__ __forceinline__ unsigned long long tbase(const IArgs& A, uint32_t p) { return 2ull * A.seg_off[p] + 64ull * p; }
__device__ __forceinline__ uint32_t tcap(const IArgs& A, uint32_t p) { return (uint32_t)(2ull * (A.seg_off[p + 1] - A.seg_off[p]) + 64ull); }
__device__ __forceinline__ unsigned long long ebase(const IArgs& A, uint32_t p) { return 16ull * A.seg_off[p] + 2048ull * p; }
__device__ __forceinline__ uint32_t ecap(const IArgs& A, uint32_t p) { return (uint32_t)(8ull * (A.seg_off[p + 1] - A.seg_off[p]) + 1024ull); }

__device__ __forceinline__ void load_consts(IrtConst* dst, uint32_t* row) {
    for (int k = threadIdx.x; k < (int)(sizeof(IrtConst) / 4); k += blockDim.x)
        reinterpret_cast<uint32_t*>(dst)[k] = reinterpret_cast<const uint32_t*>(&c_irt)[k];
    __syncthreads();
    if (threadIdx.x < 6) {
        uint32_t r = 0;             // reaction index of (s, q) in 4-bit fields, 15 = none
        for (int q = 5; q >= 0; --q) r = (r << 4) | (uint32_t)(dst->map[threadIdx.x * 6 + q] & 15);
        row[threadIdx.x] = r;
    }
    __syncthreads();
}

// 1) load + thermalisation displacement (:475-537) and species lists; W warps per track,
//    each taking a contiguous part of its entries.  What bounds it is the chain of
//    Philox blocks and f64 sums of an entry's displacement (18 draws), one chunk of 32 after
//    another; with several warps a first look at the codes alone tells where each warp's
//    particles and list entries go.
//    One warp per track took 0.37 ms for a track of 3060 entries and 0.53 ms for 4096
//    tracks of 10 keV, 8 warps 0.05 and 0.43.
template <int W>
__global__ void __launch_bounds__(W == 1 ? IB : 32 * W) k_irt_load(const __grid_constant__ IArgs A) {
    __shared__ IrtConst s_c;
    __shared__ uint32_t s_row[6], s_cnt[W][8], s_track, s_ext;
    load_consts(&s_c, s_row);
    const IrtConst& C = s_c;
    const int lane = threadIdx.x & 31, wg = W == 1 ? 0 : threadIdx.x >> 5;
    const unsigned lt = (1u << lane) - 1u;
    const uint32_t k0 = A.k0, k1 = A.k1;
    unsigned long long n_tracks = 0, n_part = 0;
    for (;;) {
        uint32_t p = 0;
        if (W == 1) {
            if (lane == 0) p = atomicAdd(&A.counters[0], 1u);
            p = __shfl_sync(FULL, p, 0);
        } else {
            if (threadIdx.x == 0) { s_track = atomicAdd(&A.counters[0], 1u); s_ext = 0; }
            __syncthreads();
            p = s_track;
        }
        if (p >= A.nseg) break;
        const unsigned long long s0 = A.seg_off[p], e0 = A.seg_off[p + 1];
        const uint32_t pid = A.pid_base + p;
        const uint32_t cap = tcap(A, p);
        const unsigned long long tb0 = tbase(A, p);
        double* px = A.px + tb0; double* py = A.py + tb0; double* pz = A.pz + tb0; double* tb = A.tb + tb0;
        int8_t* sp = A.sp + tb0; uint8_t* alive = A.alive + tb0;
        uint16_t* lst = A.lst + 6 * tb0; uint16_t* lpos = A.lpos + tb0;
        float4* rec = A.rec + 6 * tb0;
        float4* pf = A.pf + tb0;
        // particles, H2 markers and list entries before this warp's
        uint32_t n = 0, h2 = 0, cnt[6] = {0, 0, 0, 0, 0, 0};
        unsigned long long s = s0, e = e0;
        if (W > 1) {
            const unsigned long long part = (e0 - s0 + 32 * W - 1) / (32 * W) * 32;
            s = min(e0, s0 + wg * part);
            e = min(e0, s + part);
            for (unsigned long long c = s; c < e; c += 32) {
                const int code = c + lane < e ? (int)rintf(A.rad[c + lane].w) % 8 : -1;
                n += __popc(__ballot_sync(FULL, code >= 0 && code != 4 && code != 7));
                h2 += __popc(__ballot_sync(FULL, code == 7));
#pragma unroll
                for (int q = 0; q < 6; ++q)
                    cnt[q] += __popc(__ballot_sync(FULL, q == 1 ? code == 1 || code == 5 : q == 5 ? code == 6 : q != 4 && code == q));
            }
            if (lane == 0) {
                s_cnt[wg][6] = n; s_cnt[wg][7] = h2;
#pragma unroll
                for (int q = 0; q < 6; ++q) s_cnt[wg][q] = cnt[q];
            }
            __syncthreads();
            uint32_t before = 0;
            if (lane < 8)
                for (int w = 0; w < wg; ++w) before += s_cnt[w][lane];
            n = __shfl_sync(FULL, before, 6);
            h2 = __shfl_sync(FULL, before, 7);
#pragma unroll
            for (int q = 0; q < 6; ++q) cnt[q] = __shfl_sync(FULL, before, q);
        }
        // origin of the track's f32 shadow coordinates: its first rad_buf entry
        const float4 r0 = s0 < e0 ? A.rad[s0] : make_float4(0.f, 0.f, 0.f, 0.f);
        const double ox = r0.x, oy = r0.y, oz = r0.z;
        float mext = 0.0f;
        for (unsigned long long c = s; c < e; c += 32) {
            unsigned long long idx = c + lane;
            bool valid = idx < e;
            int code = -1;
            float4 r = make_float4(0.f, 0.f, 0.f, 0.f);
            if (valid) { r = A.rad[idx]; code = (int)rintf(r.w) % 8; }
            bool keep = valid && code >= 0 && code != 4 && code != 7;
            h2 += __popc(__ballot_sync(FULL, valid && code == 7));
            unsigned m = __ballot_sync(FULL, keep);
            uint32_t k = n + __popc(m & lt);
            int spc = -1;
            float4 sh = make_float4(0.f, 0.f, 0.f, 0.f);           // shadow and birth time 0
            if (keep) {
                double x = r.x, y = r.y, z = r.z;
                spc = code;
                double sigma = 0;
                int disp = 0;
                uint32_t blk = 0, wi = 4;
                u4 wb = {0, 0, 0, 0};
                auto nextd = [&]() -> double {
                    if (wi == 4) { wb = philox(blk++, k, pid, 2u, k0, k1); wi = 0; }
                    uint32_t a_ = wi == 0 ? wb.x : wb.z;
                    uint32_t b_ = wi == 0 ? wb.y : wb.w;
                    wi += 2;
                    return u01d(a_, b_);
                };
                if (code == 5) spc = 1;
                else if (code == 0 || code == 3) { if (nextd() < 0.5) { disp = 1; sigma = C.sig_oh; } }
                else if (code == 1) { disp = 1; sigma = C.sig_eaq; }
                else if (code == 2) { disp = 1; sigma = C.sig_h; }
                else if (code == 6) spc = 5;
                if (disp) {
                    double c6[3];
                    for (int ax = 0; ax < 3; ++ax) {
                        double r1 = nextd(), r2 = nextd(), r3 = nextd(), r4 = nextd(), r5 = nextd(), r6 = nextd();
                        c6[ax] = (r1 + r2 + r3 + r4 + r5 + r6 - 3) * 1.4142135623730951;
                    }
                    x += sigma * c6[0]; y += sigma * c6[1]; z += sigma * c6[2];
                }
                px[k] = x; py[k] = y; pz[k] = z; tb[k] = 0.0;
                sp[k] = (int8_t)spc; alive[k] = 1;
                float fx = (float)(x - ox), fy = (float)(y - oy), fz = (float)(z - oz);
                pf[k] = make_float4(fx, fy, fz, __int_as_float(spc));
                sh = make_float4(fx, fy, fz, 0.0f);
                mext = fmaxf(mext, fmaxf(fabsf(fx), fmaxf(fabsf(fy), fabsf(fz))));
            }
            n += __popc(m);
#pragma unroll
            for (int q = 0; q < 6; ++q) {
                const unsigned mq = __ballot_sync(FULL, spc == q);
                if (spc == q) {
                    const uint32_t at = cnt[q] + __popc(mq & lt);
                    lst[q * cap + at] = (uint16_t)k;
                    rec[q * cap + at] = sh;
                    lpos[k] = (uint16_t)at;
                }
                cnt[q] += __popc(mq);
            }
        }
        for (int o = 16; o; o >>= 1) mext = fmaxf(mext, __shfl_xor_sync(FULL, mext, o));
        if (W > 1) {
            if (lane == 0) atomicMax(&s_ext, __float_as_uint(mext));
            __syncthreads();
            mext = __uint_as_float(s_ext);
            __syncthreads();                               // read by all
            if (wg != W - 1) continue;                     // the last warp's counts are the track's
        }
        if (lane == 0) {
            A.tn[p] = n;
            A.th2[p] = h2;
            // |f32 shadow distance - f64 distance| <= 3.1e-7 * extent; 1e-6 * extent + 1e-4 nm bounds it
            A.tdel[p] = mext * 1e-6f + 1e-4f;
            uint32_t tiles = 0;                    // the pairing kernel's tiles: 32 particles of one species
#pragma unroll
            for (int q = 0; q < 6; ++q) { A.tlc[6 * p + q] = cnt[q]; tiles += (cnt[q] + 31) / 32; }
            A.ttiles[p] = tiles;
            A.tev[p] = 0;
        }
        if (n) { n_tracks++; n_part += n; }
        if (lane == 0 && n) atomicMax(&A.counters[3], n);
    }
    if (lane == 0 && n_tracks) { atomicAdd(&A.acc[12], n_tracks); atomicAdd(&A.acc[13], n_part); }
}

__device__ __forceinline__ u4 philox_accept(uint32_t blk, uint32_t i, uint32_t pid, const uint32_t* rk) {
    return philox_rk(blk, i, pid, 3u, rk);
}

// 2) initial pairing (:539-558): one warp per (track, tile of 32 particles of one
//    species).  What bounds it is the number of instructions per pair: every
//    pair inside R_CUT needs its own Philox word (4 partners to a block), so
//    everything else is kept off the pair.  The tile's particles sit in lane
//    registers; 32 partners at a time are staged in shared memory with the
//    constants of their reaction with the tile's species (a tile of one
//    species needs one table row), and those that cannot react with it, or do
//    not exist, are staged so far away that no test passes.  A pair is a
//    candidate when
//      R_CUT may hold and (U, r) may pass the exact test r2 <= R^2 of r_acc.
//    With R = max(s, s c / U) + add (times 1 + 1e-6, plus 1e-6) and the shadow
//    distance within del of the exact one, that is
//      r <= (s + add)(1+1e-6) + 1e-6 + del             (rare: `ta2`), or
//      (r - kb) U <= s c (1+1e-6)^2,  kb = add (1+1e-6) + 1e-6 + del,
//    which holds for any lower bound of U as well: the word's upper 16 bits,
//    which cost a byte permute instead of a conversion and admit 1 % more
//    candidates.  Both sides are squared, with a 1e-4 margin for the f32
//    arithmetic.  Each lane keeps its candidates in its own column of shared memory
//    (no vote per pair); a full column makes the warp pack all columns and
//    evaluate them exactly in f64, 32 at a time, one per lane.
//    The distances, the bound's products and the counts' sums run two to an
//    instruction (f32x2: one issue slot for both).
//    In a track wider than R_CUT, chunks of 32 partners whose box lies beyond it
//    from the tile's are passed by before their first pair.
//    Measured at 4096 x 10 keV: 8.1 ms, of which the scan is 4.6, SamplePDC 2.8; 8.2 ms
//    without the boxes (2048 x 30 keV 15.4 without them, 10.6 with), 9.1 ms also with
//    every SamplePDC pair through pdc_find at once, 9.5 ms also without f32x2, 10.5 ms also
//    with the rare f64 erfcx inline (the instruction cache, as in the event kernel), 14.9 ms
//    also with tiles in index order, one table gather per pair and queue votes per
//    partner (5, 6 blocks per SM: 8.5, 8.1 ms; 4, 7 were slower before the boxes).
constexpr int QCAP = 16;                 // candidates per lane
constexpr float FAR = 1e18f;             // shadow coordinate of a partner that cannot react

// two f32 values in a register pair; the packed instructions take one issue slot for both
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float a, float b) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void unpack2(f32x2 v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

__device__ __forceinline__ float warp_min(float v) {
    float r;
    asm volatile("redux.sync.min.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}
__device__ __forceinline__ float warp_max(float v) {
    float r;
    asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}

struct InitTrack {
    const double *px, *py, *pz;
    const float4* pf;
    const int8_t* sp;
    double* ET;
    uint32_t* EAB;
    uint32_t* tev;
    uint32_t ecp, pid, p;
    float lo2;                           // shadow distance^2 below which a pair is certainly inside R_CUT
};

// a warp's SamplePDC pairs: b, (i, j), track, and reaction | kinds | trial
constexpr int PDC_WAIT = 12, PDC_KEEP = 26, PDC_FEW = 20;
constexpr uint32_t PDC_Q = 96;
struct PdcQueue {
    double b[PDC_Q], lb[32];             // lb: of the pairs in the lanes
    uint32_t ij[PDC_Q], p[PDC_Q], kt[PDC_Q];
};

// exact evaluation of queued candidates [0, cnt), one per lane; returns the
// reactive pairs inside R_CUT found among those within rounding of it.  SamplePDC's pairs
// join the warp's queue Q (room for 32).
__device__ __forceinline__ uint32_t init_batch(const IrtConst& C, const InitTrack& T, const uint32_t* qij, int cnt,
                                               int lane, const uint32_t* rk, bool& ev_over, PdcQueue& Q, uint32_t& qn) {
    const unsigned lt = (1u << lane) - 1u;
    bool acc = false, pdcq = false;
    double t = 0, pa = 1, pb = 1;
    uint32_t i = 0, j = 0, np = 0, kinds = 0;
    if (lane < cnt) {
        const uint32_t ij = qij[lane];
        i = ij >> 16; j = ij & 0xffffu;
        const float4 a = T.pf[i], q = T.pf[j];
        const int si = __float_as_int(a.w), sj = __float_as_int(q.w);
        const int ri = C.map[si * 6 + sj];
        const float fx = a.x - q.x, fy = a.y - q.y, fz = a.z - q.z;
        const bool sure = fmaf(fz, fz, fmaf(fy, fy, fx * fx)) < T.lo2;     // counted by the scan
        const double dx = T.px[i] - T.px[j], dy = T.py[i] - T.py[j], dz = T.pz[i] - T.pz[j];
        const double r2 = dx * dx + dy * dy + dz * dz;
        const bool inside = sure || r2 <= C.r_cut2;
        if (inside) {
            if (!sure) np = 1;
            const u4 w4 = philox_accept(j >> 2, i, T.pid, rk);
            const double U = u01d32((j & 3) == 0 ? w4.x : (j & 3) == 1 ? w4.y : (j & 3) == 2 ? w4.z : w4.w);
            const double R = r_acc(C, ri, U);
            if (r2 <= R * R) {
                const double D = C.D[si] + C.D[sj];
                t = sample_pre(C, sqrt(r2), ri, D, U, &pa, &pb);
                if (t == -2.0) { pdcq = true; kinds = (uint32_t)(ri | si << 4 | sj << 8); }
                else acc = (t >= 0 && t < 1000);
            }
        }
    }
    const unsigned pm = __ballot_sync(FULL, pdcq);
    if (pm) {
        if (pdcq) {
            const uint32_t at = qn + __popc(pm & lt);
            Q.b[at] = pb; Q.ij[at] = (i << 16) | j; Q.p[at] = T.p; Q.kt[at] = kinds;
        }
        qn += __popc(pm);
        __syncwarp();
    }
    const unsigned m = __ballot_sync(FULL, acc);
    if (m) {
        uint32_t base = 0;
        if (lane == 0) base = atomicAdd(T.tev, (uint32_t)__popc(m));
        base = __shfl_sync(FULL, base, 0);
        const uint32_t slot = base + __popc(m & lt);
        if (acc) {
            if (slot < T.ecp) { T.ET[slot] = t; T.EAB[slot] = (i << 16) | j; }
            else ev_over = true;
        }
    }
    return np;
}

// SamplePDC of the queued pairs, a pair to a lane: every lane goes through its own
// pair's trials in order, all of them needed (pdc_find evaluates 42 % more), until
// PDC_WAIT lanes have one that passes the upper bound; these take the bracket and their
// pair's end together, and idle lanes take the next pairs.  The queue must not be empty.
// With `all` false, what is left when the queue is empty and less than PDC_KEEP lanes have a
// pair goes back to the queue, with its place in the trials; otherwise the last PDC_FEW
// pairs go through pdc_find, whose rounds are 32 trials of one pair: a few pairs need
// thousands of trials.
// Measured (pairing kernel, ms, every pair through pdc_find and this): 4096 tracks of 10 keV
// 9.05 and 8.24, 4096 of 1 keV 0.78 and 0.61, 64 of 10 keV 0.42 and 0.31; PDC_WAIT 8, 12,
// 16: 8.30, 8.24, 8.33; PDC_FEW 6, 12, 20: 64 tracks 0.64, 0.40, 0.36.
__device__ __forceinline__ void pdc_queue(const IArgs& A, const IrtConst& C, PdcQueue& Q, uint32_t& qn, bool all, int lane,
                                          bool& ev_over) {
    const unsigned lt = (1u << lane) - 1u;
    bool act = false, pend = false;
    uint32_t ij = 0, p = 0, kinds = 0, trial = 0;
    PdcPair P = {};
    u4 w = {0, 0, 0, 0};
    float hpq = 0, qpq = 0;
    auto event = [&](uint32_t wx, uint32_t wy) {
        const double X = pdc_x(C.a_pdc[kinds & 15u], Q.lb[lane], P.pq, P.M, wx, wy);
        if (!(X > 0)) return;
        const double t = X / (C.D[kinds >> 4 & 15u] + C.D[kinds >> 8]);
        if (!(t < 1000)) return;
        const uint32_t slot = atomicAdd(&A.tev[p], 1u);
        if (slot < ecap(A, p)) { A.ev_t[ebase(A, p) + slot] = t; A.ev_ab[ebase(A, p) + slot] = ij; }
        else ev_over = true;
    };
    for (;;) {
        const unsigned idle = __ballot_sync(FULL, !act);
        if (idle && qn) {
            const uint32_t take = min((uint32_t)__popc(idle), qn), rank = __popc(idle & lt);
            if (!act && rank < take) {
                const uint32_t at = qn - 1 - rank;
                ij = Q.ij[at]; p = Q.p[at];
                kinds = Q.kt[at] & 0xfffu; trial = Q.kt[at] >> 12;
                const double b = Q.b[at];
                Q.lb[lane] = b;
                P = pdc_pair(C.a_pdc[kinds & 15u], b);
                hpq = 0.5f * P.pqf; qpq = __fdividef(0.5f * P.pqf, P.Mf);
                act = true;
            }
            qn -= take;
            __syncwarp();
        }
        unsigned run = __ballot_sync(FULL, act);
        if (!run) break;
        if (qn == 0 && !all && __popc(run) < PDC_KEEP) {
            if (act) {
                const uint32_t at = __popc(run & lt);
                Q.b[at] = Q.lb[lane]; Q.ij[at] = ij; Q.p[at] = p; Q.kt[at] = kinds | trial << 12;
            }
            qn = __popc(run);
            __syncwarp();
            break;
        }
        if (qn == 0 && __popc(run) <= PDC_FEW) {
            do {
                const int src = __ffs(run) - 1;
                run &= run - 1;
                const uint32_t pid = A.pid_base + __shfl_sync(FULL, p, src);
                const double a = C.a_pdc[kinds & 15u], b = Q.lb[lane];
                const uint64_t wd = pdc_find(src, ij >> 16, ij & 0xffffu, pid, P, a, b, lane, A.rk, __shfl_sync(FULL, trial, src));
                if (lane == src && wd != ~0ull) event((uint32_t)(wd >> 32), (uint32_t)wd);
            } while (run);
            break;
        }
        // trials until enough lanes wait
        int waiting = 0;
#pragma unroll 1
        do {
            if (act && !pend) {
                w = philox_rk(ij >> 16, ij & 0xffffu, A.pid_base + p, 4u | (trial << 4), A.rk);
                pend = pdc_maybe(w, P.thr, hpq, qpq, P.Mf, P.t2f, P.af, P.bf);
                if (!pend && ++trial == 10000) act = false;
            }
            waiting = __popc(__ballot_sync(FULL, pend));
            run = __ballot_sync(FULL, act && !pend);
        } while (run && waiting < PDC_WAIT && waiting + __popc(run) > PDC_FEW);
        if (pend) {
            int st = pdc_bracket(w, P.thr, P.pqf, P.Mf, P.t2f, P.bbf, P.af, P.bf);
            if (st == 2) st = pdc_exact(w, C.a_pdc[kinds & 15u], Q.lb[lane]) ? 1 : 0;
            if (st == 1) { event(w.x, w.y); act = false; }
            else if (++trial == 10000) act = false;
            pend = false;
        }
    }
}

__global__ void __launch_bounds__(IB, 6) k_irt_init(const __grid_constant__ IArgs A) {
    __shared__ IrtConst s_c;
    __shared__ uint32_t s_row[6];
    // partners of a chunk: negated shadow x, y, z and the bound's kb and fk (scaled to 16-bit U)
    __shared__ __align__(16) float s_p[IB / 32][5][32];
    __shared__ float s_box[IB / 32][6];
    __shared__ uint16_t s_q[IB / 32][QCAP][32];
    __shared__ uint32_t s_d[IB / 32][QCAP * 32 + 32];
    __shared__ PdcQueue s_pdc[IB / 32];
    load_consts(&s_c, s_row);
    const IrtConst& C = s_c;
    const int lane = threadIdx.x & 31, wl = threadIdx.x >> 5;
    const unsigned long long nitems = A.toff[A.nseg];
    const float rcut = (float)sqrt(C.r_cut2);
    float (*sp)[32] = s_p[wl];
    float* box = s_box[wl];
    uint32_t* dq = s_d[wl];
    unsigned long long n_pairs = 0;
    uint32_t qn = 0;
    bool ev_over = false;
    for (;;) {
        unsigned long long item = 0;
        if (lane == 0) item = atomicAdd(&A.counters[1], 1u);
        item = __shfl_sync(FULL, item, 0);
        if (item >= nitems) break;
        uint32_t lo = 0, hi = A.nseg;                 // last p with toff[p] <= item
        while (hi - lo > 1) { uint32_t mid = (lo + hi) >> 1; if (A.toff[mid] <= item) lo = mid; else hi = mid; }
        const uint32_t p = lo;
        const uint32_t n = A.tn[p];
        // the item's species and its place in that species' list
        uint32_t tile = (uint32_t)(item - A.toff[p]), len = 0;
        int s = 0;
        for (; s < 6; ++s) {
            len = A.tlc[6 * p + s];
            const uint32_t nt = (len + 31) / 32;
            if (tile < nt) break;
            tile -= nt;
        }
        if (s == 6) break;                            // not reached: ttiles is the sum of these
        const uint32_t row = s_row[s];
        const unsigned long long tb0 = tbase(A, p);
        const uint32_t cap = tcap(A, p);
        const float4* pf = A.pf + tb0;
        const float del = A.tdel[p];
        const float clo = (rcut - del) * 0.99999f, chi = (rcut + del) * 1.00001f;
        const float lo2 = clo * clo, hi2 = chi * chi, lo2s = lo2 * 0x1p100f, hi2s = hi2 * 0x1p100f;
        const InitTrack T{A.px + tb0, A.py + tb0, A.pz + tb0, pf, A.sp + tb0, A.ev_t + ebase(A, p), A.ev_ab + ebase(A, p),
                          &A.tev[p], ecap(A, p), A.pid_base + p, p, lo2};
        const uint32_t at = 32u * tile + lane;
        const bool have = at < len;
        const uint32_t i = have ? A.lst[6 * tb0 + (size_t)s * cap + at] : 0xffffu;
        float4 me = make_float4(-3.0f * FAR, 0.f, 0.f, 0.f);
        if (have) me = A.rec[6 * tb0 + (size_t)s * cap + at];
        const f32x2 mx = pack2(me.x, me.x), my = pack2(me.y, me.y), mz = pack2(me.z, me.z);
        float ta2 = 0.0f;                             // (r_acc's radius for U -> 1)^2, over the row's reactions
        for (int q = 0; q < 6; ++q) {
            const int r = (int)((row >> (4 * q)) & 15u);
            if (r != 15) { const float ta = (C.fa0[r] + del) * 1.000001f; ta2 = fmaxf(ta2, ta * ta * 1.0001f); }
        }
        const uint32_t imin = __shfl_sync(FULL, i, 0);
        const uint32_t imax = __shfl_sync(FULL, i, min(31u, len - 32u * tile - 1u));
        // a track that fits into R_CUT needs no boxes (del bounds its extent)
        const bool wide = (del - 1e-4f) * 3.5e6f > rcut;
        if (wide) {                                   // the tile's box
            const float x0 = warp_min(have ? me.x : FAR), x1 = warp_max(have ? me.x : -FAR);
            const float y0 = warp_min(have ? me.y : FAR), y1 = warp_max(have ? me.y : -FAR);
            const float z0 = warp_min(have ? me.z : FAR), z1 = warp_max(have ? me.z : -FAR);
            if (lane == 0) { box[0] = x0; box[1] = x1; box[2] = y0; box[3] = y1; box[4] = z0; box[5] = z1; }
        }
        uint32_t cnt = 0, rem = 0;
        float np = 0.0f;                              // at most 32,735 partners: exact
        const uint32_t gend = (n + 3) >> 2;           // groups of 4 partners = one Philox block
        for (uint32_t g = (imin >> 5) << 3; g < gend; ++g) {
            if ((g & 7u) == 0) {
                for (;;) {
                    __syncwarp();
                    const uint32_t j = 4 * g + lane;
                    float4 q = make_float4(FAR, 0.f, 0.f, 0.f);
                    float kb = 0.0f, fk = 0.0f;
                    bool re = false;
                    if (j < n) {
                        q = pf[j];
                        const int r = (int)((row >> (4 * __float_as_int(q.w))) & 15u);
                        re = r != 15;
                        if (!re) q.x = FAR;
                        else { kb = (C.fkb0[r] + del) * 1.00006f; fk = C.fk[r] * (65536.0f * 1.00006f); }
                    }
                    // in a track wider than R_CUT, chunks of which no pair is inside it are passed by
                    // (but for the last, of which nothing comes)
                    if (wide && g + 8 < gend) {
                        // the chunk's box against the tile's: with the pairs' own operations in
                        // their order (each is monotonic), so that it holds for every pair's r2
                        const float gx = fmaxf(warp_min(re ? q.x : FAR) - box[1], box[0] - warp_max(re ? q.x : -FAR));
                        const float gy = fmaxf(warp_min(re ? q.y : FAR) - box[3], box[2] - warp_max(re ? q.y : -FAR));
                        const float gz = fmaxf(warp_min(re ? q.z : FAR) - box[5], box[4] - warp_max(re ? q.z : -FAR));
                        const float cx = fmaxf(gx, 0.0f), cy = fmaxf(gy, 0.0f), cz = fmaxf(gz, 0.0f);
                        if (fmaf(cz, cz, fmaf(cy, cy, cx * cx)) > hi2) { g += 8; continue; }
                    }
                    sp[0][lane] = -q.x; sp[1][lane] = -q.y; sp[2][lane] = -q.z; sp[3][lane] = kb; sp[4][lane] = fk;
                    __syncwarp();
                    break;
                }
            }
            const uint32_t k = (g & 7u) * 4u;
            const ulonglong2 X = *reinterpret_cast<const ulonglong2*>(&sp[0][k]), Y = *reinterpret_cast<const ulonglong2*>(&sp[1][k]);
            const ulonglong2 Z = *reinterpret_cast<const ulonglong2*>(&sp[2][k]);
            float r2[4];
            {
                const f32x2 x0 = add2(mx, X.x), y0 = add2(my, Y.x), z0 = add2(mz, Z.x);
                const f32x2 x1 = add2(mx, X.y), y1 = add2(my, Y.y), z1 = add2(mz, Z.y);
                unpack2(fma2(z0, z0, fma2(y0, y0, mul2(x0, x0))), r2[0], r2[1]);
                unpack2(fma2(z1, z1, fma2(y1, y1, mul2(x1, x1))), r2[2], r2[3]);
            }
            if (4 * g <= imax) {                      // partners not after i do not count
#pragma unroll
                for (int u = 0; u < 4; ++u) r2[u] = 4 * g + u > i ? r2[u] : FAR * FAR;
            }
            // pairs surely inside R_CUT, and those that may be: sums of saturated
            // differences (the sign decides, 2^100 makes any difference 1), which run on the
            // FP32 pipe; a compare and a count would each take two cycles of the integer one
            float lo4[4], hi4[4], nlo, nhi, nl1, nh1;
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                lo4[u] = __saturatef(fmaf(r2[u], -0x1p100f, lo2s));
                hi4[u] = __saturatef(fmaf(r2[u], -0x1p100f, hi2s));
            }
            unpack2(add2(pack2(lo4[0], lo4[1]), pack2(lo4[2], lo4[3])), nlo, nl1);
            unpack2(add2(pack2(hi4[0], hi4[1]), pack2(hi4[2], hi4[3])), nhi, nh1);
            nlo += nl1;
            nhi += nh1;
            if (nhi > 0.0f) {
                const ulonglong2 KB = *reinterpret_cast<const ulonglong2*>(&sp[3][k]), FK = *reinterpret_cast<const ulonglong2*>(&sp[4][k]);
                const u4 cw = philox_accept(g, i, T.pid, A.rk);
                const uint32_t wd[4] = {cw.x, cw.y, cw.z, cw.w};
                np += nlo;
                float v[4], uw[4];
                // 2^23 + the word's upper 16 bits, minus 2^23
#pragma unroll
                for (int u = 0; u < 4; ++u) uw[u] = __uint_as_float(__byte_perm(wd[u], 0x4B000000u, 0x7632));
#pragma unroll
                for (int u = 0; u < 4; u += 2) {
                    const f32x2 uf = add2(pack2(uw[u], uw[u + 1]), pack2(-8388608.0f, -8388608.0f));
                    float ra, rb, wa, wb;
                    unpack2(fma2(u ? KB.y : KB.x, uf, u ? FK.y : FK.x), ra, rb);
                    unpack2(mul2(pack2(r2[u], r2[u + 1]), mul2(uf, uf)), wa, wb);
                    v[u] = fmaf(ra, ra, -wa);
                    v[u + 1] = fmaf(rb, rb, -wb);
                }
                const float mn = fminf(fminf(fminf(r2[0], r2[1]), r2[2]), r2[3]);
                if (fmaxf(fmaxf(fmaxf(v[0], v[1]), v[2]), v[3]) >= 0.0f || nhi != nlo || mn <= ta2) {
#pragma unroll
                    for (int u = 0; u < 4; ++u)
                        if ((v[u] >= 0.0f || !(r2[u] < lo2) || r2[u] <= ta2) && r2[u] <= hi2) {
                            s_q[wl][cnt][lane] = (uint16_t)(4 * g + u);
                            cnt++;
                        }
                }
            }
            const bool last = g + 1 == gend;
            if (last || __any_sync(FULL, cnt > QCAP - 4)) {
                __syncwarp();
                uint32_t off = cnt;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) { const uint32_t v = __shfl_up_sync(FULL, off, o); if (lane >= o) off += v; }
                const uint32_t total = rem + __shfl_sync(FULL, off, 31);
                off += rem - cnt;
                for (uint32_t c = 0; c < cnt; ++c) dq[off + c] = (i << 16) | s_q[wl][c][lane];
                cnt = 0;
                __syncwarp();
                uint32_t b = 0;
                for (; b + (last ? 1u : 32u) <= total; b += 32) {
                    n_pairs += init_batch(C, T, dq + b, (int)min(32u, total - b), lane, A.rk, ev_over, s_pdc[wl], qn);
                    if (qn > PDC_Q - 32) pdc_queue(A, C, s_pdc[wl], qn, false, lane, ev_over);
                }
                rem = 0;
                if (b < total) {
                    rem = total - b;
                    const uint32_t v = (uint32_t)lane < rem ? dq[b + lane] : 0u;
                    __syncwarp();
                    if ((uint32_t)lane < rem) dq[lane] = v;
                }
                __syncwarp();
            }
        }
        n_pairs += (unsigned long long)np;
    }
    if (qn) pdc_queue(A, C, s_pdc[wl], qn, true, lane, ev_over);
    if (__any_sync(FULL, ev_over) && lane == 0) atomicOr(A.err, DERR_HEAP);
    for (int o = 16; o; o >>= 1) n_pairs += __shfl_xor_sync(FULL, n_pairs, o);
    if (lane == 0 && n_pairs) atomicAdd(&A.acc[10], n_pairs);
}

// 3) the initial events of each track in (t, i, j) order (:566): a block-wide
//     bitonic sort, in shared memory up to SORT_SM events (padded to a power
//     of two).  A larger track is cut into chunks that blocks of their own sort
//     (k_irt_sort_chunks) and merge by rank into the second half of the track's event slots
//     (they hold 2 ecap; k_irt_sort_merge): one block's bitonic sort of 16,626 events in
//     global memory took 2.2 ms, bound by one SM's latency, this 0.06 ms.  These two
//     kernels cost a launch each even when no track needs them, so they run only when
//     tracks are long enough to have that many events as a rule (sort_chunked); a dense
//     track below that is sorted in its slots by its one block.
//     Keys are unique, so the order is that of any other sort.
constexpr int SB = 256;
constexpr uint32_t SORT_SM = 4096;
constexpr int SCB = 512;
constexpr uint32_t SORT_CH = 2048;       // events per chunk
__device__ __forceinline__ bool sort_chunked(const IArgs& A, uint32_t nev) { return nev > SORT_SM && A.pcap > IRT_PCAP_MIN; }
__global__ void __launch_bounds__(SB) k_irt_sort(IArgs A) {
    __shared__ double st[SORT_SM];
    __shared__ uint32_t sab[SORT_SM];
    for (uint32_t k = blockIdx.x; k < A.nseg; k += gridDim.x) {
        const uint32_t p = A.order[k];                 // largest tracks first
        const uint32_t nev = A.tev[p];
        if (nev < 2 || nev > ecap(A, p)) continue;     // the event kernel reports the overflow
        double* T = A.ev_t + ebase(A, p);
        uint32_t* AB = A.ev_ab + ebase(A, p);
        uint32_t n2 = 2;
        while (n2 < nev) n2 <<= 1;
        if (sort_chunked(A, nev)) {
            const uint32_t nch = (nev + SORT_CH - 1) / SORT_CH;
            if (threadIdx.x == 0) {
                const uint32_t at = atomicAdd(&A.counters[4], nch);
                for (uint32_t c = 0; c < nch; ++c) A.big[at + c] = (unsigned long long)p << 32 | c;
            }
            continue;
        }
        const bool sm = n2 <= SORT_SM;
        double* t = sm ? st : T;
        uint32_t* ab = sm ? sab : AB;
        __syncthreads();                               // the previous track is written back
        for (uint32_t i = threadIdx.x; i < n2; i += SB) {
            if (i >= nev) { t[i] = 1e300; ab[i] = 0xffffffffu; }
            else if (sm) { st[i] = T[i]; sab[i] = AB[i]; }
        }
        __syncthreads();
        for (uint32_t kk = 2; kk <= n2; kk <<= 1) {
            for (uint32_t j = kk >> 1; j > 0; j >>= 1) {
                for (uint32_t q = threadIdx.x; q < (n2 >> 1); q += SB) {
                    const uint32_t i = ((q & ~(j - 1)) << 1) | (q & (j - 1)), l = i | j;   // bit j of i clear
                    const double ti = t[i], tl = t[l];
                    const uint32_t ai = ab[i], al = ab[l];
                    if (ev_less(tl, al, ti, ai) == ((i & kk) == 0)) { t[i] = tl; t[l] = ti; ab[i] = al; ab[l] = ai; }
                }
                __syncthreads();
            }
        }
        if (sm)
            for (uint32_t i = threadIdx.x; i < nev; i += SB) { T[i] = st[i]; AB[i] = sab[i]; }
    }
}

__global__ void __launch_bounds__(SCB) k_irt_sort_chunks(const __grid_constant__ IArgs A) {
    __shared__ double st[SORT_CH];
    __shared__ uint32_t sab[SORT_CH];
    const uint32_t n = A.counters[4];
    for (uint32_t k = blockIdx.x; k < n; k += gridDim.x) {
        const uint32_t p = (uint32_t)(A.big[k] >> 32), c = (uint32_t)A.big[k];
        double* T = A.ev_t + ebase(A, p) + c * SORT_CH;
        uint32_t* AB = A.ev_ab + ebase(A, p) + c * SORT_CH;
        const uint32_t len = min(SORT_CH, A.tev[p] - c * SORT_CH);
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < SORT_CH; i += SCB) {
            st[i] = i < len ? T[i] : 1e300;
            sab[i] = i < len ? AB[i] : 0xffffffffu;
        }
        __syncthreads();
        for (uint32_t kk = 2; kk <= SORT_CH; kk <<= 1)
            for (uint32_t j = kk >> 1; j > 0; j >>= 1) {
#pragma unroll
                for (uint32_t q0 = 0; q0 < SORT_CH / 2; q0 += SCB) {
                    const uint32_t q = q0 + threadIdx.x;
                    const uint32_t i = ((q & ~(j - 1)) << 1) | (q & (j - 1)), l = i | j;   // bit j of i clear
                    const double ti = st[i], tl = st[l];
                    const uint32_t ai = sab[i], al = sab[l];
                    if (ev_less(tl, al, ti, ai) == ((i & kk) == 0)) { st[i] = tl; st[l] = ti; sab[i] = al; sab[l] = ai; }
                }
                __syncthreads();
            }
        for (uint32_t i = threadIdx.x; i < len; i += SCB) { T[i] = st[i]; AB[i] = sab[i]; }
    }
}

// an event's place: its place in its chunk plus the events before it in the track's others
__global__ void __launch_bounds__(SB) k_irt_sort_merge(const __grid_constant__ IArgs A) {
    __shared__ double st[SORT_CH];
    __shared__ uint32_t sab[SORT_CH];
    constexpr uint32_t PARTS = SORT_CH / SB;
    const uint32_t n = A.counters[4] * PARTS;
    for (uint32_t k = blockIdx.x; k < n; k += gridDim.x) {
        const unsigned long long e = A.big[k / PARTS];
        const uint32_t p = (uint32_t)(e >> 32), c = (uint32_t)e, nev = A.tev[p];
        double* T = A.ev_t + ebase(A, p);
        uint32_t* AB = A.ev_ab + ebase(A, p);
        const uint32_t i = c * SORT_CH + k % PARTS * SB + threadIdx.x;
        if (i - threadIdx.x >= nev) continue;
        const bool have = i < nev;
        const double t = have ? T[i] : 0.0;
        const uint32_t ab = have ? AB[i] : 0u;
        uint32_t pos = i - c * SORT_CH;
        for (uint32_t d = 0; d * SORT_CH < nev; ++d) {
            if (d == c) continue;
            const uint32_t len = min(SORT_CH, nev - d * SORT_CH);
            __syncthreads();
            for (uint32_t q = threadIdx.x; q < len; q += SB) { st[q] = T[d * SORT_CH + q]; sab[q] = AB[d * SORT_CH + q]; }
            __syncthreads();
            uint32_t lo = 0, hi = len;
            while (lo < hi) {
                const uint32_t m = (lo + hi) >> 1;
                if (ev_less(st[m], sab[m], t, ab)) lo = m + 1; else hi = m;
            }
            pos += lo;
        }
        if (have) { T[ecap(A, p) + pos] = t; AB[ecap(A, p) + pos] = ab; }
    }
}

__device__ __forceinline__ double gauss_axis(uint32_t wa, uint32_t wb) {
    return sqrt(-2 * log_(u01d32(wa) + 1e-30)) * cos_(6.2831853 * u01d32(wb));
}
__device__ __forceinline__ float sqrt_fast(float x) {                // 2^-22 relative; 0 below 2^-126
    float r;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float log2_fast(float x) {                // 2^-22 absolute in [1/2, 2], relative outside
    float r;
    asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

template <int B>
__device__ __forceinline__ void cp_async(void* dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "n"(B)
                 : "memory");
}
template <int N>
__device__ __forceinline__ void cp_wait() {                          // this lane's copies but the last N, seen by the warp
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
    __syncwarp();
}

// 4) events (:566-660): pop the sorted initial events in (t, i, j) order merged
//    with a heap of product events; W warps per track.  The first warp pops
//    (stale events and reactions without products change nothing the others work on);
//    a product is re-paired with the alive partners of the species that react
//    with it (pairWithAlive, :430-465) in three steps over all lanes of the W warps:
//    an f32 scan that lists the partners it cannot rule out, their exact f64
//    evaluation, and the accepted events' way into the heap.
//
// What bounds it: with few tracks, a track's chain of events, one after another, so W
// grows as the tracks get fewer (loop_width).  With many, fetching instructions: the
// kernel's code is far larger than the SM's instruction cache and the warps are at
// different places in it (a third of the fetches missed; at 16 warps per SM 5.6 of 11.5
// cycles between a warp's instructions were that, and 28 warps were no faster).  So
// the rare f64 paths are out of line and rolled, one copy of the scan serves all species,
// and at W = 1 the four tracks of a block go from one re-pairing to the next together.
// The rest keeps work off the chain:
// * initial events come in windows of 32, copied to shared memory ahead; a window's events
//   whose species are dead are dropped at once, and a reaction drops those of its two;
// * kind and life of each species are in shared memory (state), 4 bits each;
// * the scan's first test bounds the partner's displacement from the product of its
//   three radius draws (one logarithm); the second runs on full warps of what is left;
// * in the exact step the three axes of a partner's Gaussian (the longest f64
//   chains) run on three lanes;
// * accepted events are written behind the heap's last node by all lanes.
// Measured (ms, before and after): 4096 tracks of 10 keV 20.0 -> 14.0, 64 of them 6.7 ->
// 2.7, 4096 of 1 keV 2.2 -> 1.53, one track of 3060 species 17.5 -> 6.1.  Before: one
// warp per track, events popped by one lane against states in global memory, a binary heap,
// batches of 64 listed partners.
constexpr int WN = 4;                    // windows of initial events in shared memory
constexpr int CQ = 128;                  // listed partners in shared memory, the rest in global
// heap nodes and species whose state is in shared memory
template <int W>
constexpr int HS = W >= 4 ? 1024 : 256 * W;
template <int W>
constexpr uint32_t SN = W >= 8 ? 16640 : 8192;
template <int W>
struct EvGroup {
    double tl[35], ht[HS<W>], wt[WN][32], et;
    unsigned long long cnt[12];          // reactions 0..8, reacted, events, initial events
    uint32_t hab[HS<W>], cq[CQ], wab[WN][32], eab, track, ncand, nacc, hn;
    int lc[6], have, si, sj, ri;
    uint32_t state[SN<W> / 8];           // 4 bits per species: kind, and 8 while it is alive
    uint32_t nq[W][64];                  // per warp: partners the first test leaves (place in the list | reaction | species)
    uint8_t src[W][32];                  // per warp: lanes that need a Gaussian
    uint8_t wsp[32];                     // kinds of a window's species
};

// The scan's f32 tests of a partner (list record q): false only if the exact step
// would reject it.
struct ScanP {
    float x, y, z, del, et, dtm, rcut;   // the product's shadow and birth time
    uint32_t id, pid;
};
// First without draws: the displacement is at most the largest Box-Muller radius of
// 32-bit draws (sqrt(3 * 2 ln 2^33) = 11.72) times sqrt(2 D dt), and a partner beyond
// R_CUT after it is rejected by the exact path too (a quarter of them, 10 keV).  Then
// with the radius of the three draws, against R of the acceptance draw: one in 18 is
// left.  dth: upper bound of dt = et - t_birth from the f32 birth time (error < dtm).
__device__ __forceinline__ bool scan_near(const ScanP& P, const float4& q, uint32_t jj, float Djf2, float fs, float fsc,
                                          float fadd, const uint32_t* rk) {
    const float ex = P.x - q.x, ey = P.y - q.y, ez = P.z - q.z;
    const float dlo = (sqrt_fast(fmaf(ez, ez, fmaf(ey, ey, ex * ex))) - P.del) * 0.999997f;
    const float dth = fmaxf(P.et - q.w + P.dtm, 0.0f);
    const float sg = sqrt_fast(Djf2 * dth) * 1.00001f;
    const bool far = dlo - sg * 11.8f > P.rcut;             // (no branch: some lane goes on in 9 of 10 chunks)
    const u4 q0 = philox_rk(P.id, jj, P.pid, 5u, rk);
    // -2 ln u summed over the axes is -2 ln of the product (>= 2^-99; the sum to 1.4e-6
    // absolute, so its root to 2e-3)
    const float u0 = u01f32(q0.x), u1 = u01f32(q0.y), u2 = u01f32(q0.z);
    const float Bm = sqrt_fast(fmaxf(-1.3864330f * log2_fast(u0 * u1 * u2), 0.0f)) + 2e-3f;
    // beyond R = max(fs, fsc / U) + fadd of r_acc, for U >= uf, times 1.00002 plus 1e-6
    const float uf = __uint2float_rd(q0.w) * 2.3283064365386963e-10f;
    const float d = fmaf(-sg, Bm, dlo) * 0.99998f - fadd - 1e-6f;
    return !(far || (d > fs && d * uf > fsc));
}
// Second: the partner displaced by the same draws in f32.
__device__ __forceinline__ bool scan_maybe(const ScanP& P, const float4& q, uint32_t jj, float Djf2, float fs, float fsc,
                                           float fadd, const uint32_t* rk) {
    const float ex = P.x - q.x, ey = P.y - q.y, ez = P.z - q.z;
    const float dth = P.et - q.w + P.dtm;
    const float sg = dth > 0.0f ? sqrt_fast(Djf2 * dth) * 1.00001f : 0.0f;
    const u4 q0 = philox_rk(P.id, jj, P.pid, 5u, rk), q1 = philox_rk(P.id, jj, P.pid, 5u | (1u << 4), rk);
    const float uf = __uint2float_rd(q0.w) * 2.3283064365386963e-10f;
    const float rhi = (fmaxf(fs, __fdividef(fsc, uf)) + fadd) * 1.00002f + 1e-6f;
    // per axis |g_f - g| <= 2e-3 + 2e-5 |g| (sqrt of the log near 0, fast log and cos, 2
    // ulp each), sigma within [sl, sg]
    const float dtl = fmaxf(P.et - q.w - P.dtm, 0.0f);
    const float sl = sqrt_fast(Djf2 * dtl) * 0.99999f, sm = 0.5f * (sg + sl);
    const float r0 = fmaxf(-2.0f * __logf(u01f32(q0.x)), 0.0f), r1 = fmaxf(-2.0f * __logf(u01f32(q0.y)), 0.0f),
                r2 = fmaxf(-2.0f * __logf(u01f32(q0.z)), 0.0f);
    const float Bm = sqrt_fast(r0 + r1 + r2) * 1.0001f + 2e-3f;
    // cos(2 pi u) = -cos(2 pi (u - 1/2)): the argument stays in [-pi, pi]
    const float g0 = -sqrt_fast(r0) * __cosf(6.2831853f * (u01f32(q1.x) - 0.5f));
    const float g1 = -sqrt_fast(r1) * __cosf(6.2831853f * (u01f32(q1.y) - 0.5f));
    const float g2 = -sqrt_fast(r2) * __cosf(6.2831853f * (u01f32(q1.z) - 0.5f));
    const float fx = ex - g0 * sm, fy = ey - g1 * sm, fz = ez - g2 * sm;
    const float d2 = sqrt_fast(fmaf(fz, fz, fmaf(fy, fy, fx * fx)));
    const float eg = 2e-3f + 2e-5f * Bm;
    const float err = 1.7320508f * (sg * eg + 0.5f * (Bm + eg) * (sg - sl)) + P.del;
    return !(dth > 0.0f) || !((d2 - err) * 0.99999f > rhi);
}

// Exact pairWithAlive step (:430-465) for listed partners, at most one per lane (e; on:
// this lane has one): Brownian sync of the partner by sqrt(2 D_j dt), R_CUT, then
// sampleIRT.  Returns whether the pair reacts, at *ta.
__device__ __forceinline__ bool pair_exact(const IArgs& A, const IrtConst& C, unsigned long long tb0, uint32_t id, uint32_t pid,
                                double Di, uint32_t e, bool on, int lane, uint8_t* src, double* ta) {
    const uint32_t* rk = A.rk;
    bool acc = false, pdcq = false, gs = false;
    double pa = 1, pb = 1, pD = 1, sig = 0, xj = 0, yj = 0, zj = 0, Dj = 0;
    const double pet = A.tb[tb0 + id];
    const uint32_t jj = e & 0xffffu;
    const int r2i = (int)((e >> 16) & 15u), s2 = (int)(e >> 20);
    u4 q0 = {0, 0, 0, 0}, q1 = {0, 0, 0, 0};
    if (on) {
        Dj = C.D[s2];
        const double dt = pet - A.tb[tb0 + jj];
        xj = A.px[tb0 + jj]; yj = A.py[tb0 + jj]; zj = A.pz[tb0 + jj];
        q0 = philox_rk(id, jj, pid, 5u, rk);
        q1 = philox_rk(id, jj, pid, 5u | (1u << 4), rk);
        gs = dt > 0;
        if (gs) sig = sqrt(2.0 * Dj * dt);
    }
    const double U = u01d32(q0.w);
    // the Gaussians: ten partners at a time, lane 3 k + a takes axis a of the k-th
    const unsigned gm = __ballot_sync(FULL, gs);
    if (gm) {
        const int rank = __popc(gm & ((1u << lane) - 1u)), ng = __popc(gm), a = lane % 3;
        if (gs) src[rank] = (uint8_t)lane;
        __syncwarp();
#pragma unroll 1
        for (int b = 0; b < ng; b += 10) {
            const int k = b + lane / 3, from = src[min(k, ng - 1)];
            const uint32_t w0 = __shfl_sync(FULL, q0.x, from), w1 = __shfl_sync(FULL, q0.y, from), w2 = __shfl_sync(FULL, q0.z, from);
            const uint32_t v0 = __shfl_sync(FULL, q1.x, from), v1 = __shfl_sync(FULL, q1.y, from), v2 = __shfl_sync(FULL, q1.z, from);
            double g = 0;
            if (k < ng && lane < 30) g = gauss_axis(a == 0 ? w0 : a == 1 ? w1 : w2, a == 0 ? v0 : a == 1 ? v1 : v2);
            const int at = 3 * (rank - b);
            const bool mine = gs && rank >= b && rank < b + 10;
            const double g0 = __shfl_sync(FULL, g, mine ? at : 0), g1 = __shfl_sync(FULL, g, mine ? at + 1 : 0);
            const double g2 = __shfl_sync(FULL, g, mine ? at + 2 : 0);
            if (mine) { xj += g0 * sig; yj += g1 * sig; zj += g2 * sig; }
        }
        __syncwarp();
    }
    if (on) {
        const double dx = A.px[tb0 + id] - xj, dy = A.py[tb0 + id] - yj, dz = A.pz[tb0 + id] - zj;
        const double r2 = dx * dx + dy * dy + dz * dz;
        if (r2 <= C.r_cut2) {
            const double D = Di + Dj;
            const double t = sample_pre(C, sqrt(r2), r2i, D, U, &pa, &pb);
            if (t == -2.0) { pdcq = true; pD = D; }
            else if (t >= 0) { *ta = pet + t; acc = *ta < 1000; }
        }
    }
    unsigned pm = __ballot_sync(FULL, pdcq);
    if (pm) {
        const PdcPair PP = pdc_pair(pa, pb);
        uint64_t words = ~0ull;
        while (pm) {
            const int s = __ffs(pm) - 1;
            pm &= pm - 1;
            const uint64_t wd = pdc_find(s, id, jj, pid, PP, pa, pb, lane, rk);
            if (lane == s) words = wd;
        }
        if (pdcq && words != ~0ull) {
            const double X = pdc_x(pa, pb, PP.pq, PP.M, (uint32_t)(words >> 32), (uint32_t)words);
            if (X > 0) { *ta = pet + X / pD; acc = *ta < 1000; }
        }
    }
    return acc;
}

template <int W>
constexpr int LT = W <= 4 ? IB : 32 * W;    // 16 warps per SM

// One meeting of the block's IB threads, which come to it at different places of the kernel
// (__syncthreads_count asks for one place, or one condition); how many came with `more`.
__device__ __forceinline__ uint32_t block_meet(bool more) {
    uint32_t n;
    __syncwarp();
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %1, 0;\n\tbarrier.red.popc.u32 %0, 1, %2, p;\n\t}"
                 : "=r"(n)
                 : "r"((uint32_t)more), "n"(IB)
                 : "memory");
    return n;
}

template <int W>
__global__ void __launch_bounds__(LT<W>, 512 / LT<W>) k_irt_loop(const __grid_constant__ IArgs A) {
    constexpr int G = LT<W> / 32 / W;            // tracks per block
    __shared__ EvGroup<W> s_g[G];
    __shared__ IrtConst s_c;
    __shared__ uint32_t s_row[6];
    load_consts(&s_c, s_row);
    const IrtConst& C = s_c;
    const int lane = threadIdx.x & 31, wg = (threadIdx.x >> 5) % W, g = (threadIdx.x >> 5) / W;
    const bool lead = wg == 0 && lane == 0;
    EvGroup<W>& S = s_g[g];
    auto gsync = [g]() {
        __syncwarp();
        if (W > 1) asm volatile("barrier.sync %0, %1;" ::"r"(1 + g), "n"(32 * W) : "memory");
    };
    const uint32_t gw = blockIdx.x * G + g;
    // CAP of the reference worker (:405): twice the largest track's species, plus 512
    const uint32_t capref = 2u * A.counters[3] + 512u;
    for (int k = lane + 32 * wg; k < 35; k += 32 * W) S.tl[k] = 0.0;
    for (int k = lane + 32 * wg; k < 12; k += 32 * W) S.cnt[k] = 0;
    // global storage of the group: heap beyond HS, partners beyond CQ
    uint32_t* gab = A.hov_ab + (size_t)gw * (A.hcap + A.pcap);
    uint32_t* gcq = gab + A.hcap;
    Heap<HS<W>> H{S.ht, S.hab, A.hov_t + (size_t)gw * A.hcap, gab};
    unsigned long long n_pairs = 0;
    for (;;) {
        if (lead) S.track = atomicAdd(&A.counters[2], 1u);
        gsync();
        const uint32_t k = S.track;
        gsync();
        if (k >= A.nseg) break;
        const uint32_t p = A.order[k];                 // largest tracks first
        const uint32_t n = A.tn[p];
        if (n == 0) continue;
        const uint32_t pid = A.pid_base + p;
        const uint32_t cap = tcap(A, p);
        const unsigned long long tb0 = tbase(A, p), eb0 = ebase(A, p) + (sort_chunked(A, A.tev[p]) ? ecap(A, p) : 0u);
        const uint32_t nev = A.tev[p];
        const float del = A.tdel[p];
        const float4 org = A.rad[A.seg_off[p]];
        if (nev > ecap(A, p)) { if (lead) atomicOr(A.err, DERR_HEAP); continue; }
        if (wg == 0 && lane < 6) S.lc[lane] = (int)A.tlc[6 * p + lane];     // alive species of each kind
        if (lead) { S.cnt[11] += nev; S.cnt[10] += nev; }
        // the state of each species in shared memory, or in global memory in tracks too large for it
        const bool insm = cap <= SN<W>;
        if (insm) {
            for (uint32_t k8 = lane + 32 * wg; k8 < (cap + 7) / 8; k8 += 32 * W) {
                uint32_t v = 0;
#pragma unroll
                for (uint32_t q = 0; q < 8; ++q) {
                    const uint32_t k1 = 8 * k8 + q;
                    if (k1 < n) v |= (uint32_t)(A.sp[tb0 + k1] | 8) << (4 * q);
                }
                S.state[k8] = v;
            }
            gsync();
        }
        auto state = [&](uint32_t k1) -> uint32_t {
            return insm ? S.state[k1 >> 3] >> (4 * (k1 & 7)) & 15u
                        : (uint32_t)A.sp[tb0 + k1] | (A.alive[tb0 + k1] ? 8u : 0u);
        };
        __syncwarp();
        // the first warp takes the initial events by windows of 32; wlive marks those whose
        // two species are alive, and the next windows are copied to shared memory ahead
        uint32_t ip = 0, hn = 0, ntot = n, wlive = 0;
        auto window = [&](uint32_t at) {
            if (at + lane < nev) {
                cp_async<8>(&S.wt[at / 32 % WN][lane], A.ev_t + eb0 + at + lane);
                cp_async<4>(&S.wab[at / 32 % WN][lane], A.ev_ab + eb0 + at + lane);
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
        if (wg == 0)
#pragma unroll 1
            for (int w = 0; w < WN - 1; ++w) window(32 * w);
        double h2c = (double)A.th2[p];
        int cp = 0, c16 = 0;
        float* curve = A.curves ? A.curves + 80ull * p : nullptr;
        bool heap_over = false;
        for (;;) {
            if (wg == 0) {
                // pop until a reaction with products
                int have = 0;
                for (;;) {
                    while (!wlive && ip < nev) {           // the next window: its live events
                        cp_wait<WN - 2>();
                        const bool in = ip + lane < nev;
                        const uint32_t wab = S.wab[ip / 32 % WN][lane], wi = wab >> 16, wj = wab & 0xffffu;
                        const uint32_t ws = in ? state(wi) | state(wj) << 4 : 0u;
                        S.wsp[lane] = (uint8_t)(ws & 0x77u);
                        wlive = __ballot_sync(FULL, (ws & 0x88u) == 0x88u);
                        ip += 32;
                        window(ip + 32 * (WN - 2));
                        __syncwarp();
                    }
                    const bool hi_ = wlive != 0, hh = hn > 0;
                    if (!hi_ && !hh) break;
                    const int w = hi_ ? __ffs(wlive) - 1 : 0;
                    const int wb = (ip / 32 + WN - 1) % WN;
                    const double ti = S.wt[wb][w], th = hh ? S.ht[0] : 0.0;
                    const uint32_t ai = S.wab[wb][w], ah = hh ? S.hab[0] : 0u;
                    const int spi = S.wsp[w];
                    const bool init = hi_ && (!hh || ev_less(ti, ai, th, ah));
                    const double et = init ? ti : th;
                    const uint32_t eab = init ? ai : ah;
                    const int ei = (int)(eab >> 16), ej = (int)(eab & 0xffffu);
                    int a = spi & 15, b2 = spi >> 4;
                    if (init) wlive &= wlive - 1;
                    else {
                        const uint32_t s0 = state(ei), s1 = state(ej);
                        a = (int)(s0 & 7u); b2 = (int)(s1 & 7u);
                        heap_pop(H, hn, lane);
                        if (!(s0 & s1 & 8u)) continue;
                    }
                    while (cp < 7 && et >= c_cp[cp]) {
                        if (lane < 5) S.tl[cp * 5 + lane] += lane == 4 ? h2c : (double)S.lc[lane == 3 ? 4 : lane];
                        cp++;
                    }
                    while (curve && c16 < 16 && et >= C.t16[c16]) {
                        if (lane < 5) curve[5 * c16 + lane] = lane == 4 ? (float)h2c : (float)S.lc[lane == 3 ? 4 : lane];
                        c16++;
                    }
                    const int r = C.map[(a < b2 ? a : b2) * 6 + (a < b2 ? b2 : a)];
                    if (r < 0) continue;
                    __syncwarp();
                    if (lane < 6) {                        // where the products will be
                        const double* at = (lane < 2 ? A.px : lane < 4 ? A.py : A.pz) + tb0 + (lane & 1 ? ej : ei);
                        asm volatile("prefetch.global.L1 [%0];" ::"l"(at));
                    }
                    // both leave their species' list (its last entry takes the place)
                    const int st = a == b2 ? 1 : 2;
                    if (lane < st) {
#pragma unroll 1
                        for (int w2 = lane; w2 < 2; w2 += st) {
                            const int k2 = w2 == 0 ? ei : ej, q = w2 == 0 ? a : b2;
                            if (insm) atomicAnd(&S.state[k2 >> 3], ~(8u << (4 * (k2 & 7))));
                            else A.alive[tb0 + k2] = 0;
                            const uint32_t at = A.lpos[tb0 + k2], end = (uint32_t)S.lc[q] - 1;
                            const uint16_t last = A.lst[6 * tb0 + q * cap + end];
                            A.rec[6 * tb0 + q * cap + at] = A.rec[6 * tb0 + q * cap + end];
                            A.lst[6 * tb0 + q * cap + at] = last;
                            A.lpos[tb0 + last] = (uint16_t)at;
                            S.lc[q] = (int)end;
                        }
                    }
                    if (lane == 0) { S.cnt[9]++; S.cnt[r]++; }
                    const uint32_t wab = S.wab[wb][lane];
                    const int wi = (int)(wab >> 16), wj = (int)(wab & 0xffffu);
                    wlive &= ~__ballot_sync(FULL, wi == ei || wi == ej || wj == ei || wj == ej);
                    __syncwarp();
                    if (r == 3 || r == 4 || r == 6) h2c += 1;
                    if (C.nprod[r] == 0) continue;
                    have = 1;
                    if (lane == 0) { S.et = et; S.eab = eab; S.si = a; S.sj = b2; S.ri = r; }
                    break;
                }
                if (lane == 0) S.have = have;
            }
            gsync();
            if (!S.have) break;
            const double et = S.et;
            const uint32_t eab = S.eab;
            const int ei = (int)(eab >> 16), ej = (int)(eab & 0xffffu);
            const int si = S.si, sj = S.sj, ri = S.ri;
            const int np_ = C.nprod[ri];
            if (W > 1) gsync();                            // all have read the event
            else block_meet(true);                         // the block's tracks go on together
#pragma unroll 1
            for (int pp = 0; pp < np_; ++pp) {
                const int nsp = pp == 0 ? C.prod0[ri] : C.prod1[ri];
                const uint32_t id = ntot;
                if (id >= capref) break;                   // the reference's CAP (:405, :621)
                if (id >= cap) { if (lead) atomicOr(A.err, DERR_TRACK_SIZE); break; }
                ntot++;
                // an axis per lane: one copy of the division
                const int ax = lane % 3;
                double* pa = (ax == 0 ? A.px : ax == 1 ? A.py : A.pz) + tb0;
                double v;
                if (np_ == 1) {                            // at the diffusion-weighted centre
                    const double sqDi = C.sqD[si], sqDj = C.sqD[sj];
                    v = (sqDj * pa[ei] + sqDi * pa[ej]) / (sqDi + sqDj);
                } else {                                   // at the two reactants
                    v = pa[pp == 0 ? ei : ej];
                }
                const double nx = __shfl_sync(FULL, v, 0), ny = __shfl_sync(FULL, v, 1), nz = __shfl_sync(FULL, v, 2);
                if (wg == 0 && lane < 3) pa[id] = v;
                ScanP P;
                P.x = (float)(nx - (double)org.x); P.y = (float)(ny - (double)org.y); P.z = (float)(nz - (double)org.z);
                P.del = del; P.et = (float)et; P.dtm = 1e-4f + 1e-6f * P.et;
                P.rcut = (float)sqrt(C.r_cut2) * 1.00001f;
                P.id = id; P.pid = pid;
                if (lead) {
                    const int at = S.lc[nsp];
                    A.tb[tb0 + id] = et;
                    if (insm) atomicOr(&S.state[id >> 3], (8u | (uint32_t)nsp) << (4 * (id & 7)));
                    else { A.sp[tb0 + id] = (int8_t)nsp; A.alive[tb0 + id] = 1; }
                    A.lst[6 * tb0 + nsp * cap + at] = (uint16_t)id;
                    A.rec[6 * tb0 + nsp * cap + at] = make_float4(P.x, P.y, P.z, P.et);
                    A.lpos[tb0 + id] = (uint16_t)at;
                    S.lc[nsp] = at + 1;
                    S.ncand = 0; S.nacc = 0; S.hn = hn;
                }
                gsync();
                const uint32_t rowp = s_row[nsp];
                // Chunks of 32 partners, over the lists of all species that react with the product;
                // the next chunk's list entries and records are loaded before this chunk is
                // tested (the lists do not change here).  What the first test leaves waits in nq
                // until 32 can take the second.  One copy of the code serves all species and
                // the rest at the end: see the kernel's comment.
                uint32_t qn = 0, nli = 0, nlen = 0, njj = 0, ntag = 0;
                int ns2 = -1;
                float4 nrec = make_float4(0.f, 0.f, 0.f, 0.f);
                auto advance = [&]() {
#pragma unroll 1
                    while (nli - lane >= nlen) {
                        if (++ns2 == 6) return;
                        const uint32_t r2i = (rowp >> (4 * ns2)) & 15u;
                        if (r2i == 15u) continue;
                        // the product itself is the last of its own list
                        nlen = (uint32_t)S.lc[ns2] - (ns2 == nsp ? 1u : 0u);
                        nli = 32u * wg + lane;
                        ntag = (r2i << 16) | ((uint32_t)ns2 << 20);
                        if (wg == 0) n_pairs += nlen;          // (as many on every lane)
                    }
                    if (nli < nlen) {
                        const size_t at = 6 * tb0 + (uint32_t)ns2 * cap + nli;
                        nrec = A.rec[at];
                        njj = A.lst[at];
                    }
                };
                nli = lane;
                advance();
#pragma unroll 1
                for (;;) {
                    const int s2 = ns2;
                    if (s2 < 6) {
                        const float4 q = nrec;
                        const uint32_t jj = njj, at = nli, tag = ntag;
                        const bool in = at < nlen;
                        nli += 32u * W;
                        advance();
                        bool nr = false;
                        if (in) {
                            const int r2i = (int)(tag >> 16 & 15u);
                            nr = scan_near(P, q, jj, C.D2f[s2], C.fs[r2i], C.fsc[r2i], C.fadd[r2i], A.rk);
                        }
                        const unsigned m = __ballot_sync(FULL, nr);
                        if (!m) continue;
                        if (nr) S.nq[wg][qn + __popc(m & ((1u << lane) - 1u))] = at | tag;
                        qn += __popc(m);
                        __syncwarp();
                        if (qn < 32) continue;
                    }
                    if (qn) {
                        const uint32_t from = qn >= 32 ? qn - 32 : 0;
                        bool mv = false;
                        uint32_t v = 0;
                        if (from + lane < qn) {
                            const uint32_t e = S.nq[wg][from + lane];
                            const int ri2 = (int)((e >> 16) & 15u), sj2 = (int)(e >> 20);
                            const size_t at = (size_t)sj2 * cap + (e & 0xffffu);
                            const uint32_t jj = A.lst[6 * tb0 + at];
                            mv = scan_maybe(P, A.rec[6 * tb0 + at], jj, C.D2f[sj2], C.fs[ri2], C.fsc[ri2], C.fadd[ri2], A.rk);
                            v = (e & ~0xffffu) | jj;
                        }
                        qn = from;
                        const unsigned m = __ballot_sync(FULL, mv);
                        if (m) {
                            uint32_t base = 0;
                            if (lane == 0) base = atomicAdd(&S.ncand, (uint32_t)__popc(m));
                            base = __shfl_sync(FULL, base, 0);
                            if (mv) {
                                base += __popc(m & ((1u << lane) - 1u));
                                if (base < CQ) S.cq[base] = v; else gcq[base - CQ] = v;
                            }
                        }
                        __syncwarp();
                    }
                    if (s2 == 6) break;
                }
                gsync();
                const uint32_t nc = S.ncand;
                if (nc == 0) continue;
                // few partners per warp when there are several warps: their chains run side by side
                constexpr uint32_t BL = W == 1 ? 32u : 8u;
#pragma unroll 1
                for (uint32_t b = BL * wg; b < nc; b += BL * W) {
                    const bool on = (uint32_t)lane < BL && b + lane < nc;
                    const uint32_t at = b + lane;
                    const uint32_t e = on ? (at < CQ ? S.cq[at] : gcq[at - CQ]) : 0u;
                    double ta = 0;
                    const bool acc = pair_exact(A, C, tb0, id, pid, C.D[nsp], e, on, lane, S.src[wg], &ta);
                    const unsigned m = __ballot_sync(FULL, acc);
                    if (m) {
                        uint32_t base = 0;
                        if (lane == 0) base = atomicAdd(&S.nacc, (uint32_t)__popc(m));
                        base = __shfl_sync(FULL, base, 0);
                        if (acc) {
                            base += __popc(m & ((1u << lane) - 1u));
                            const uint32_t pj = e & 0xffffu;
                            base += S.hn;                  // the heap's next free nodes
                            if (base < HS<W> + A.hcap) H.set(base, ta, pj < id ? (pj << 16) | id : (id << 16) | pj);
                        }
                    }
                }
                gsync();
                if (wg == 0) {
                    const uint32_t na = S.nacc;
                    if (lane == 0) {
                        S.cnt[10] += na;
#pragma unroll 1
                        for (uint32_t q = hn; q < min(hn + na, HS<W> + A.hcap); ++q) heap_up(H, q);
                    }
                    heap_over |= hn + na > HS<W> + A.hcap;
                    hn = min(hn + na, HS<W> + A.hcap);
                    __syncwarp();
                }
            }
        }
        if (wg == 0) {
            if (heap_over && lane == 0) atomicOr(A.err, DERR_HEAP);
            if (lane < 5) {
                const double v = lane == 4 ? h2c : (double)S.lc[lane == 3 ? 4 : lane];
                for (; cp < 7; cp++) S.tl[cp * 5 + lane] += v;
                for (; curve && c16 < 16; c16++) curve[5 * c16 + lane] = (float)v;
            }
            __syncwarp();
        }
    }
    if (W == 1) while (block_meet(false)) {}               // until the block's last track has ended
    if (lane == 0 && n_pairs) atomicAdd(&A.acc[10], n_pairs);
    gsync();
    if (lead) {
        for (int k = 0; k < 10; ++k) if (S.cnt[k]) atomicAdd(&A.acc[k], S.cnt[k]);
        if (S.cnt[10]) atomicAdd(&A.acc[11], S.cnt[10]);
        if (S.cnt[11]) atomicAdd(&A.acc[14], S.cnt[11]);
    }
    for (int k = lane + 32 * wg; k < 35; k += 32 * W)
        if (S.tl[k] != 0.0) atomicAdd(&A.acc_tl[k], S.tl[k]);
}

// codes -> grouping keys (pid << 34 | original index) for a caller's rad_buf
__global__ void k_group_keys(const float4* rad, unsigned long long n, unsigned long long* key, uint32_t* maxpid) {
    unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x;
    uint32_t mp = 0;
    if (i < n) {
        int w = (int)rintf(rad[i].w);
        uint32_t pid = w >= 0 ? (uint32_t)(w / 8) : 0u;
        key[i] = ((unsigned long long)pid << 34) | i;
        mp = pid;
    }
    for (int o = 16; o; o >>= 1) mp = max(mp, __shfl_xor_sync(0xffffffffu, mp, o));
    if ((threadIdx.x & 31) == 0) atomicMax(maxpid, mp);
}

// longest segment
__global__ void k_seg_max(const unsigned long long* off, uint32_t nseg, unsigned long long* out) {
    unsigned long long m = 0;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < nseg; i += gridDim.x * blockDim.x)
        m = max(m, off[i + 1] - off[i]);
    for (int o = 16; o; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) atomicMax(out, m);
}

// ------------------------------------------------------------------ host side
cudaError_t irt_set_constants(const IrtConst& c, cudaStream_t s) {
    const cudaError_t e = cudaMemcpyToSymbolAsync(c_irt, &c, sizeof c, 0, cudaMemcpyHostToDevice, s);
    return e != cudaSuccess ? e : cudaStreamSynchronize(s);
}

static int blocks_for(const void* k, int device, uint32_t limit = 0) {
    int sms = 0, per = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k, IB, 0);
    if (per < 1) per = 1;
    if (limit && (int)limit < per) per = (int)limit;
    return sms * per;
}

// Order of the event kernel's tracks: by species count, largest first (a
// bucket sort in one block), so the longest event chains start early and the
// last wave holds the short ones.
__global__ void __launch_bounds__(1024) k_track_order(const uint32_t* tn, uint32_t nseg, uint32_t* order) {
    constexpr int NB = 512;
    __shared__ uint32_t cnt[NB], off[NB];
    __shared__ uint32_t smax;
    if (threadIdx.x == 0) smax = 0;
    for (int b = threadIdx.x; b < NB; b += blockDim.x) cnt[b] = 0;
    __syncthreads();
    uint32_t m = 0;
    for (uint32_t p = threadIdx.x; p < nseg; p += blockDim.x) m = max(m, tn[p]);
    atomicMax(&smax, m);
    __syncthreads();
    const uint32_t mx = smax > 0 ? smax : 1;
    for (uint32_t p = threadIdx.x; p < nseg; p += blockDim.x)
        atomicAdd(&cnt[(uint32_t)(((unsigned long long)(mx - min(tn[p], mx)) * (NB - 1)) / mx)], 1u);
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t a = 0;
        for (int b = 0; b < NB; ++b) { off[b] = a; a += cnt[b]; }
    }
    __syncthreads();
    for (uint32_t p = threadIdx.x; p < nseg; p += blockDim.x) {
        const uint32_t b = (uint32_t)(((unsigned long long)(mx - min(tn[p], mx)) * (NB - 1)) / mx);
        order[atomicAdd(&off[b], 1u)] = p;
    }
}

// Warps per track of the load: several where there are few tracks for the SMs, of long
// ones (over 480 entries) also with more; many tracks fill the warps by themselves.
// Measured (us, 1 and 8): 16 tracks of 10 keV 186 and 30, 592: 265 and 90, 4096: 529 and
// 430; 64 of 1 keV 40 and 18, 592: 50 and 26, 4096: 91 and 98, 16384: 221 and 370; 65,536
// of 0.1 to 30 keV 3097 and 3523.
constexpr int LOAD_W = 8;
static bool load_wide(int device, const IArgs& a) {
    int sms = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    return a.nseg <= (a.pcap > IRT_PCAP_MIN ? 64u : 4u) * (unsigned)sms;
}

// Warps per track of the event kernel: two while all tracks are resident at once at 16 warps
// per SM, more while they are at 8 per SM.  Measured (10 keV tracks on 148 SMs, ms with
// W = 1, 2, 4, 8, 16): 64 tracks 5.12 3.09 2.88 2.80 2.87, 150: 5.46 3.15 2.89 2.80 3.57,
// 300: 5.69 3.45 3.36 3.75 5.97, 600: 5.81 3.95 4.37 6.29 -, 1200: 6.39 5.63 7.39 - -,
// 1800: 7.25 8.21 10.2 - -; one track of 3060 species 7.85 6.81 6.56 6.52 6.53.
static int loop_width(int device, uint32_t nseg) {
    int sms = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    const unsigned long long warps = 16ull * (unsigned long long)sms;
    int w = 16;
    while (w > 1 && (unsigned long long)nseg * (unsigned long long)w > (w > 2 ? warps / 2 : warps)) w >>= 1;
    return w;
}

// resident blocks of the event kernel with W warps per track; the shape's limit is in
// blocks of 4 warps
template <int W>
static int loop_blocks(int device, const IrtShape& shape) {
    int sms = 0, per = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, (const void*)k_irt_loop<W>, LT<W>, 0);
    if (per < 1) per = 1;
    const int limit = (int)shape.loop_per_sm * IB / LT<W>;
    if (shape.loop_per_sm && limit < per) per = limit > 0 ? limit : 1;
    return sms * per;
}
template <int W>
static int loop_groups(int device, const IrtShape& shape) {
    return loop_blocks<W>(device, shape) * (LT<W> / 32 / W);
}

// tracks of the event kernel in flight at once, at most: each has its own scratch (asking for
// the width in use alone keeps the other widths' code from being loaded)
// (blocks hold up to 4 tracks, of which the last may be without one)
int irt_warps(int device, const IrtShape& shape, uint32_t nseg) {
    int n = 1;
    switch (loop_width(device, nseg)) {
    case 16: n = loop_groups<16>(device, shape); break;
    case 8: n = loop_groups<8>(device, shape); break;
    case 4: n = loop_groups<4>(device, shape); break;
    case 2: n = loop_groups<2>(device, shape); break;
    default: n = loop_groups<1>(device, shape);
    }
    return (int)std::min((unsigned long long)n, ((unsigned long long)nseg + 3) & ~3ull);
}

template <int W>
static cudaError_t launch_loop(const IArgs& a, int device, const IrtShape& shape, cudaStream_t s) {
    const unsigned groups = LT<W> / 32 / W, fit = (unsigned)loop_blocks<W>(device, shape);
    const unsigned want = (a.nseg + groups - 1) / groups;
    k_irt_loop<W><<<want < fit ? (want ? want : 1) : fit, LT<W>, 0, s>>>(a);
    return cudaGetLastError();
}

// tile prefix: the scan of transport.cu
cudaError_t launch_scan_u32(const uint32_t* cnt, uint32_t n, unsigned long long* off, cudaStream_t s);

// timing events of the launch sequence: inside a stream capture they must be
// external event nodes, which a replay records like a plain cudaEventRecord
static cudaError_t irt_mark(cudaEvent_t e, cudaStream_t s) {
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    cudaError_t r = cudaStreamIsCapturing(s, &cs);
    if (r != cudaSuccess) return r;
    return cudaEventRecordWithFlags(e, s, cs == cudaStreamCaptureStatusActive ? cudaEventRecordExternal
                                                                              : cudaEventRecordDefault);
}

cudaError_t launch_irt(const IArgs& a, int device, const IrtShape& shape, cudaStream_t s, cudaEvent_t* ev) {
    { cudaError_t me_ = cudaMemsetAsync(a.counters, 0, 8 * sizeof(uint32_t), s); if (me_ != cudaSuccess) return me_; }
    if (load_wide(device, a)) {
        int sms = 0;
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
        const unsigned fit = 8u * (unsigned)sms;           // at most 8 blocks of 8 warps per SM; they take tracks in turn
        k_irt_load<LOAD_W><<<a.nseg < fit ? (a.nseg ? a.nseg : 1) : fit, 32 * LOAD_W, 0, s>>>(a);
    } else {
        k_irt_load<1><<<blocks_for((const void*)k_irt_load<1>, device), IB, 0, s>>>(a);
    }
    cudaError_t e = launch_scan_u32(a.ttiles, a.nseg, a.toff, s);
    if (e != cudaSuccess) return e;
    if (ev && (e = irt_mark(ev[0], s)) != cudaSuccess) return e;
    k_irt_init<<<blocks_for((const void*)k_irt_init, device, shape.init_per_sm), IB, 0, s>>>(a);
    if (ev && (e = irt_mark(ev[1], s)) != cudaSuccess) return e;
    k_track_order<<<1, 1024, 0, s>>>(a.tn, a.nseg, a.order);
    int sms = 0, per = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, (const void*)k_irt_sort, SB, 0);
    const unsigned long long sgrid = (unsigned long long)sms * (unsigned long long)(per > 0 ? per : 1);
    k_irt_sort<<<(unsigned)(a.nseg < sgrid ? (a.nseg > 0 ? a.nseg : 1) : sgrid), SB, 0, s>>>(a);
    if (a.pcap > IRT_PCAP_MIN) {
        k_irt_sort_chunks<<<2 * sms, SCB, 0, s>>>(a);
        k_irt_sort_merge<<<4 * sms, SB, 0, s>>>(a);
    }
    if (ev && (e = irt_mark(ev[2], s)) != cudaSuccess) return e;
    switch (loop_width(device, a.nseg)) {
    case 16: return launch_loop<16>(a, device, shape, s);
    case 8: return launch_loop<8>(a, device, shape, s);
    case 4: return launch_loop<4>(a, device, shape, s);
    case 2: return launch_loop<2>(a, device, shape, s);
    default: return launch_loop<1>(a, device, shape, s);
    }
}

// The IRT launch sequence: plain launches when anything in the arguments (seed
// included) or the shapes differs from the call before; a call that repeats them
// captures the sequence as one CUDA graph, on a private stream, which further
// repetitions replay on the caller's.  Capturing for every new seed or track set cost
// each such call 0.24 ms (64 tracks of 1 keV 0.95 -> 0.71 ms with plain launches, 4096
// of 100 eV 0.55 -> 0.30, a context's first call 0.5 ms less); a replay among other host
// work saves 0.17 ms (training data of 4096 x 1 keV 5.08 -> 4.91).  If capturing fails the
// sequence runs as plain launches from then on.
cudaError_t irt_graph_run(const IArgs& a, int device, const IrtShape& shape, cudaStream_t s, cudaEvent_t* ev,
                          IrtGraph* g) {
    if (g->off) return launch_irt(a, device, shape, s, ev);
    IrtGraphKey want;
    memset(&want, 0, sizeof want);
    want.a = a;
    want.shape = shape;
    want.device = device;
    want.ev = ev;
    cudaError_t e;
    if (memcmp(&g->key, &want, sizeof want) != 0) {
        if (g->exec) { cudaGraphExecDestroy(g->exec); g->exec = nullptr; }
        memcpy(&g->key, &want, sizeof want);     // with its padding
        return launch_irt(a, device, shape, s, ev);
    }
    if (!g->exec) {
        cudaStream_t cs;
        if ((e = cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking)) != cudaSuccess) return e;
        cudaGraph_t gr = nullptr;
        e = cudaStreamBeginCapture(cs, cudaStreamCaptureModeThreadLocal);
        if (e == cudaSuccess) {
            cudaError_t le = launch_irt(a, device, shape, cs, ev);
            e = cudaStreamEndCapture(cs, &gr);
            if (le != cudaSuccess) e = le;
        }
        if (e == cudaSuccess) e = cudaGraphInstantiate(&g->exec, gr, 0);
        if (gr) cudaGraphDestroy(gr);
        cudaStreamDestroy(cs);
        if (e != cudaSuccess) {
            cudaGetLastError();                  // clear the failed capture
            g->exec = nullptr;
            g->off = true;
            return launch_irt(a, device, shape, s, ev);
        }
    }
    return cudaGraphLaunch(g->exec, s);
}

cudaError_t launch_group_keys(const float4* rad, unsigned long long n, unsigned long long* key, uint32_t* maxpid,
                              cudaStream_t s) {
    { cudaError_t me_ = cudaMemsetAsync(maxpid, 0, 4, s); if (me_ != cudaSuccess) return me_; }
    if (n) k_group_keys<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(rad, n, key, maxpid);
    return cudaGetLastError();
}

cudaError_t launch_seg_max(const unsigned long long* off, uint32_t nseg, unsigned long long* out, cudaStream_t s) {
    { cudaError_t me_ = cudaMemsetAsync(out, 0, 8, s); if (me_ != cudaSuccess) return me_; }
    k_seg_max<<<148, 256, 0, s>>>(off, nseg, out);
    return cudaGetLastError();
}

}  // namespace wg
