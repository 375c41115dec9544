// surrogate.cu -- learned chemistry for the IRT: track descriptors and a small
// MLP (64 -> 128 -> 128 -> 128 -> 80, GELU) trained and evaluated with
// hand-written tcgen05 kernels: bf16 operands in shared memory (K-major,
// no swizzle), f32 accumulators in tensor memory, one elected thread issuing
// the MMAs, an mbarrier signalled by tcgen05.commit.
//
// One CTA of 16 warps per tile of 128 tracks runs the 4 layers back to back
// and, in training, the loss and the 4 backward steps as well, with everything
// between the inputs and the weight gradients kept on the SM: layer inputs and
// their transposes (bf16) in shared memory, pre-activations and products (f32)
// in tensor memory, weights brought in by one bulk copy per layer.  Warp w owns
// TMEM lanes 32 (w % 4) .. + 31 = rows of the tile, and columns 32 (w / 4) .. + 31
// of each 128-column product, so an epilogue (bias, GELU, bf16 rounding) is 32
// values per thread.
//
// Backward: per layer, the input gradient dH = D W and the weight gradient
// dW = D^T H (K = the tile's 128 rows).  Each CTA sums the weight gradients of its
// tiles in its own slice of a partial-gradient buffer, which the optimiser adds up
// in CTA order: no atomics on the gradient.  Loss: mean squared error over the
// batch and the 80 outputs of the standardised G(t) curves.
#include "surrogate.cuh"
#include "common.cuh"

namespace wg {

// ------------------------------------------------------------ PTX helpers
__device__ __forceinline__ uint32_t s2u(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ unsigned long long sg_time() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ void mbar_init(uint64_t* b, uint32_t cnt) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(s2u(b)), "r"(cnt) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ bool mbar_try(uint64_t* b, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(s2u(b)), "r"(parity)
        : "memory");
    return ok != 0;
}

// wait for the phase of the given parity, at most lim_ns (0: give up before
// the first poll)
__device__ bool mbar_wait(uint64_t* b, uint32_t parity, unsigned long long lim_ns) {
    if (lim_ns == 0) return false;
    const unsigned long long t0 = sg_time();
    while (!mbar_try(b, parity))
        if (sg_time() - t0 > lim_ns) return false;
    return true;
}

// Wait for the MMAs committed to phase `parity`.  A wait that runs out clears
// *ok (the kernel reports SG_ERR_WAIT) and is followed by a drain wait of at
// most WG_MMA_WAIT_NS, so that tensor memory is not read, reissued or freed
// under an MMA still in flight.
__device__ __forceinline__ void mma_wait(uint64_t* b, uint32_t parity, unsigned long long lim_ns, bool& ok) {
    if (!mbar_wait(b, parity, lim_ns)) {
        ok = false;
        mbar_wait(b, parity, WG_MMA_WAIT_NS);
    }
}

// one elected thread: bring `bytes` (a multiple of 16) from global to shared
// memory and have the barrier complete when they are there
__device__ __forceinline__ void bulk_load(uint8_t* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(s2u(bar)), "r"(bytes) : "memory");
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(s2u(dst)),
                 "l"(src), "r"(bytes), "r"(s2u(bar))
                 : "memory");
}

__device__ __forceinline__ void tmem_alloc(uint32_t* dst, uint32_t ncols) {     // one full warp
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(s2u(dst)), "r"(ncols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {   // the allocating warp
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}

__device__ __forceinline__ void tc_before_sync() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_after_sync() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// all threads: make generic shared-memory writes visible to the tensor cores,
// and order earlier tensor-memory reads before later MMAs
__device__ __forceinline__ void sg_sync() {
    fence_async_smem();
    tc_before_sync();
    __syncthreads();
    tc_after_sync();
}

// Shared-memory matrix descriptor: K-major, no swizzle.  Core matrices are
// 8 rows x 16 bytes stored contiguously (128 B); the next core matrix along K
// is LBO bytes on, the next group of 8 rows SBO bytes on; version 1 (bit 46).
__device__ __forceinline__ uint64_t sdesc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
    return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
           ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}

// Instruction descriptor of kind::f16: bf16 A and B (both K-major), f32 D, M x N.
__host__ __device__ constexpr uint32_t idesc_bf16(int M, int N) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

// byte offset of element (r, k) of an R x K operand in that layout (core
// matrices packed along K: LBO 128, SBO 16 K)
__host__ __device__ __forceinline__ uint32_t coff(uint32_t r, uint32_t k, uint32_t K) {
    return ((((r >> 3) * (K >> 3)) + (k >> 3)) << 7) + ((r & 7u) << 4) + ((k & 7u) << 1);
}
// The transposed operands (K = the tile's 128 rows) are written two bytes at a
// time, 32 rows by a warp: a core-matrix stride of 144 bytes along K spreads
// the four core matrices of a warp over different banks (128 would put them all
// on the same four).
constexpr uint32_t T_LBO = 144, T_SBO = 15 * T_LBO + 128;
__device__ __forceinline__ uint32_t toff(uint32_t r, uint32_t k) {
    return (r >> 3) * T_SBO + (k >> 3) * T_LBO + ((r & 7u) << 4) + ((k & 7u) << 1);
}

__device__ __forceinline__ void umma_bf16(uint32_t d_tmem, uint64_t ad, uint64_t bd, uint32_t id, uint32_t accum) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}"
        ::"r"(d_tmem), "l"(ad), "l"(bd), "r"(id), "r"(accum), "r"(0u), "r"(0u), "r"(0u), "r"(0u)
        : "memory");
}

__device__ __forceinline__ void umma_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(s2u(bar))
                 : "memory");
}

// D (TMEM, M x N f32) = A (M x K) * B (N x K)^T, K a multiple of 16; one thread
__device__ __forceinline__ void gemm_issue(uint32_t d_tmem, uint32_t sa, uint32_t lbo_a, uint32_t sbo_a, uint32_t sb,
                                           uint32_t lbo_b, uint32_t sbo_b, int M, int N, int K) {
    const uint32_t id = idesc_bf16(M, N);
    for (int j = 0; j < K / 16; ++j)
        umma_bf16(d_tmem, sdesc(sa + 2u * lbo_a * j, lbo_a, sbo_a), sdesc(sb + 2u * lbo_b * j, lbo_b, sbo_b), id,
                  j > 0 ? 1u : 0u);
}

// 32 consecutive f32 columns of this warp's 32 TMEM lanes (one row per thread)
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float* v) {
    uint32_t r[32];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(r[j]);
}

// the reverse: 32 columns of the warp's lanes from registers
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const float* v) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
        ::"r"(taddr), "r"(__float_as_uint(v[0])), "r"(__float_as_uint(v[1])), "r"(__float_as_uint(v[2])), "r"(__float_as_uint(v[3])), "r"(__float_as_uint(v[4])), "r"(__float_as_uint(v[5])), "r"(__float_as_uint(v[6])), "r"(__float_as_uint(v[7])),
        "r"(__float_as_uint(v[8])), "r"(__float_as_uint(v[9])), "r"(__float_as_uint(v[10])), "r"(__float_as_uint(v[11])), "r"(__float_as_uint(v[12])), "r"(__float_as_uint(v[13])), "r"(__float_as_uint(v[14])), "r"(__float_as_uint(v[15])),
        "r"(__float_as_uint(v[16])), "r"(__float_as_uint(v[17])), "r"(__float_as_uint(v[18])), "r"(__float_as_uint(v[19])), "r"(__float_as_uint(v[20])), "r"(__float_as_uint(v[21])), "r"(__float_as_uint(v[22])), "r"(__float_as_uint(v[23])),
        "r"(__float_as_uint(v[24])), "r"(__float_as_uint(v[25])), "r"(__float_as_uint(v[26])), "r"(__float_as_uint(v[27])), "r"(__float_as_uint(v[28])), "r"(__float_as_uint(v[29])), "r"(__float_as_uint(v[30])), "r"(__float_as_uint(v[31]))
        : "memory");
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

// GELU and its derivative from one error function
__device__ __forceinline__ float gelu(float z, float* deriv) {
    const float e = 1.0f + erff(z * 0.70710678118654752f);
    if (deriv) *deriv = 0.5f * e + z * 0.39894228040143268f * __expf(-0.5f * z * z);
    return 0.5f * z * e;
}

constexpr uint32_t SG_ERR_WAIT = 1u << 6;    // an mbarrier wait gave up

// Column sums of a warp's 32 x 32 values (row = lane): lane c gets column c.
// Halving exchange, 31 shuffles; the sums associate as an xor butterfly's
// from 16 down to 1.
__device__ __forceinline__ float colsum32(float* v, int lane) {
#pragma unroll
    for (int o = 16; o; o >>= 1) {
#pragma unroll
        for (int k = 0; k < o; ++k) {
            const bool up = (lane & o) != 0;
            const float keep = up ? v[k + o] : v[k], send = up ? v[k] : v[k + o];
            v[k] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
    }
    return v[0];
}

// one row's `cnt` (a multiple of 8, at most 32) values from column c0 on into a K-major operand
__device__ __forceinline__ void put_row(uint8_t* dst, int row, int c0, uint32_t K, const __nv_bfloat16* h, int cnt) {
#pragma unroll
    for (int c = 0; c < 4; ++c)
        if (8 * c < cnt) *reinterpret_cast<uint4*>(dst + coff(row, c0 + 8 * c, K)) = *reinterpret_cast<const uint4*>(h + 8 * c);
}
// and into a transposed operand
__device__ __forceinline__ void put_col(uint8_t* dst, int row, int c0, const __nv_bfloat16* h, int cnt) {
#pragma unroll
    for (int j = 0; j < 32; ++j)
        if (j < cnt) *reinterpret_cast<__nv_bfloat16*>(dst + toff(c0 + j, row)) = h[j];
}

constexpr int SG_THREADS = 512;
constexpr uint32_t SG_BUF = 32768;                              // a 128 x 128 bf16 operand
constexpr uint32_t SG_TBUF = 16 * T_SBO;                        // a transposed one
// training: A operand (H or D), weights, D^T, H1^T, H2^T, H3^T, H0^T (64 rows)
constexpr uint32_t SG_SMEM_TRAIN = 2 * SG_BUF + 4 * SG_TBUF + SG_TBUF / 2;
constexpr uint32_t SG_SMEM_FWD = 2 * SG_BUF;

// What bounds it: the chain of 4 (training: 11) products, each one MMA issue, one
// wait and one epilogue, on as many SMs as the batch has tiles (8 at the recipe's
// 1024 rows).  16 warps share an epilogue, the next weights are copied while it
// runs, and the whole step is one launch beside the optimiser's.
// Measured per step of 1024 rows (two launches): 1580 us with forward and backward
// kernels of 4 warps that passed activations through global memory, added every
// bias gradient to one shared word and every weight gradient to one global one;
// 47 us now, 44.5 of them this kernel (forward alone 96 -> 17 us).
template <bool TRAIN>
__global__ void __launch_bounds__(SG_THREADS, 1) k_sg(SgArgs a) {
    extern __shared__ __align__(128) uint8_t sm[];
    uint8_t* bufA = sm;
    uint8_t* bufW = sm + SG_BUF;
    uint8_t* bufGT = sm + 2 * SG_BUF;                           // TRAIN only, like HT
    uint8_t* HT[4] = {bufGT + 4 * SG_TBUF, bufGT + SG_TBUF, bufGT + 2 * SG_TBUF, bufGT + 3 * SG_TBUF};
    __shared__ uint64_t bar, bar_w;
    __shared__ uint32_t tbase;
    __shared__ float sdb[TRAIN ? 4 : 1][SG_HID];                // column sums of D by 32 rows
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int row = 32 * (warp & 3) + lane, c0 = 32 * (warp >> 2);
    constexpr uint32_t NCOL = TRAIN ? 512 : 128;
    // TMEM: pre-activations (then their gelu') of layers 1..3, then the region of outputs and input gradients
    constexpr uint32_t REG = TRAIN ? 384 : 0;
    if (warp == 0) tmem_alloc(&tbase, NCOL);
    if (tid == 0) { mbar_init(&bar, 1); mbar_init(&bar_w, 1); }
    sg_sync();
    const uint32_t tm = tbase, lane_tm = tm + ((uint32_t)(32 * (warp & 3)) << 16);
    bool ok = true;
    uint32_t ph = 0, wph = 0;
    const int OFFB[4] = {SG_OFF_B1, SG_OFF_B2, SG_OFF_B3, SG_OFF_B4};
    const int OFFW[4] = {SG_OFF_W1, SG_OFF_W2, SG_OFF_W3, SG_OFF_W4};
    const uint32_t ntiles = (a.n + SG_TILE - 1) / SG_TILE;
    for (uint32_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        if (tid == 0) bulk_load(bufW, a.w.W[0], SG_HID * SG_IN * 2, &bar_w);
        const uint32_t r = tile * SG_TILE + row;
        const bool live = r < a.n;
        const uint32_t src = live ? (a.rows ? a.rows[r] : r) : 0u;
        {   // input row -> bf16, 16 columns per thread
            const int k0 = 16 * (warp >> 2);
            __align__(16) __nv_bfloat16 h[16];
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const float4 q = live ? reinterpret_cast<const float4*>(a.X + (size_t)src * SG_IN + k0)[c]
                                      : make_float4(0.f, 0.f, 0.f, 0.f);
                float x[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int k = k0 + 4 * c + j;
                    if (a.xmean && live) x[j] = (x[j] - a.xmean[k]) * a.xinv[k];
                    h[4 * c + j] = __float2bfloat16_rn(x[j]);
                }
            }
            put_row(bufA, row, k0, SG_IN, h, 16);
            if (TRAIN) put_col(HT[0], row, k0, h, 16);
        }
        sg_sync();
#pragma unroll
        for (int l = 0; l < 4; ++l) {
            const int K = l == 0 ? SG_IN : SG_HID, N = l == 3 ? SG_OUT : SG_HID;
            const uint32_t reg = TRAIN ? 128u * l : 0u;         // layer 3: REG
            if (tid == 0) {
                mma_wait(&bar_w, wph & 1u, a.mma_ns, ok);
                gemm_issue(tm + reg, s2u(bufA), 128u, 16u * K, s2u(bufW), 128u, 16u * K, SG_TILE, N, K);
                umma_commit(&bar);
            }
            wph++;
            mma_wait(&bar, ph & 1u, (l == 0 && a.give_up_first) ? 0ull : a.mma_ns, ok);
            ph++;
            tc_after_sync();
            if (tid == 0) {                                     // the weights are read: bring the next ones
                if (l < 3) bulk_load(bufW, a.w.W[l < 3 ? l + 1 : 3], (l == 2 ? SG_OUT : SG_HID) * SG_HID * 2, &bar_w);
                else if (TRAIN) bulk_load(bufW, a.w.WT[3], SG_OUT * SG_HID * 2, &bar_w);
            }
            const float* bias = a.w.p + OFFB[l];
            if (c0 < N) {
                float v[32];
                tmem_ld32(lane_tm + reg + (uint32_t)c0, v);
                if (l < 3) {
                    __align__(16) __nv_bfloat16 h[32];
#pragma unroll
                    for (int j = 0; j < 32; ++j)
                        h[j] = __float2bfloat16_rn(gelu(v[j] + bias[c0 + j], TRAIN ? &v[j] : nullptr));
                    put_row(bufA, row, c0, SG_HID, h, 32);
                    if (TRAIN) {
                        put_col(HT[l + 1], row, c0, h, 32);
                        tmem_st32(lane_tm + reg + (uint32_t)c0, v);   // gelu'(Z) in Z's place
                    }
                } else if (!TRAIN) {
                    const int cnt = min(32, SG_OUT - c0);
                    if (a.Y && live) {
                        float* y = a.Y + (size_t)r * SG_OUT + c0;
#pragma unroll
                        for (int j = 0; j < 32; j += 4)
                            if (j < cnt) {
                                float o[4];
#pragma unroll
                                for (int k = 0; k < 4; ++k)
                                    o[k] = (v[j + k] + bias[c0 + j + k]) * a.ystd[c0 + j + k] + a.ymean[c0 + j + k];
                                *reinterpret_cast<float4*>(y + j) = make_float4(o[0], o[1], o[2], o[3]);
                            }
                    }
                    if (a.acc) {
                        // column sums over the tile's rows: each warp adds its 32
                        // rows in f32, then its partial in f64
                        const float e = live ? (a.E ? a.E[r] : a.E0) : 0.0f;
#pragma unroll
                        for (int j = 0; j < 32; ++j)
                            v[j] = live && j < cnt ? ((v[j] + bias[c0 + j]) * a.ystd[c0 + j] + a.ymean[c0 + j]) * e : 0.0f;
                        const float w = colsum32(v, lane);
                        if (lane < cnt) atomicAdd(&a.acc[c0 + lane], (double)w);
                        if (c0 == 0) {
                            float w2 = e;
#pragma unroll
                            for (int o = 16; o; o >>= 1) w2 += __shfl_xor_sync(0xffffffffu, w2, o);
                            if (lane == 0) atomicAdd(&a.acc[SG_OUT], (double)w2);
                        }
                    }
                } else {
                    // D_3 = dL/dY = 2 (Y - T) / (n * 80); rows past n contribute zeros
                    const int cnt = min(32, SG_OUT - c0);
                    const float scale = 2.0f / ((float)a.n * (float)SG_OUT);
                    double sse = 0.0;
                    __align__(16) __nv_bfloat16 h[32];
#pragma unroll
                    for (int j = 0; j < 32; ++j) {
                        float d = 0.0f;
                        if (live && j < cnt) {
                            d = (v[j] + bias[c0 + j]) - a.T[(size_t)src * SG_OUT + c0 + j];
                            sse += (double)d * d;
                        }
                        v[j] = d * scale;
                        h[j] = __float2bfloat16_rn(v[j]);
                    }
                    for (int o = 16; o; o >>= 1) sse += __shfl_xor_sync(0xffffffffu, sse, o);
                    if (lane == 0 && sse != 0.0) atomicAdd(a.loss, sse);
                    put_row(bufA, row, c0, SG_OUT, h, cnt);
                    put_col(bufGT, row, c0, h, cnt);
                    const float w = colsum32(v, lane);
                    if (lane < cnt) sdb[TRAIN ? warp & 3 : 0][c0 + lane] = w;
                }
            }
            sg_sync();
        }
        if (TRAIN) {
            float* part = a.part + (size_t)blockIdx.x * SG_NPARAM;
            const bool first = tile == blockIdx.x;
#pragma unroll
            for (int l = 3; l >= 0; --l) {
                const int n_out = l == 3 ? SG_OUT : SG_HID, n_in = l == 0 ? SG_IN : SG_HID;
                // bias gradient of this layer: the column sums of D_l
                if (tid < n_out) {
                    float* b = part + OFFB[l] + tid;
                    float w = 0.0f;
#pragma unroll
                    for (int q = 0; q < (TRAIN ? 4 : 1); ++q) w += sdb[q][tid];
                    *b = first ? w : *b + w;
                }
                float d[32];
                if (l > 0) {
                    // dH_l, then D_{l-1} = dH_l gelu'(Z_l) in registers
                    if (tid == 0) {
                        mma_wait(&bar_w, wph & 1u, a.mma_ns, ok);
                        gemm_issue(tm + REG, s2u(bufA), 128u, 16u * n_out, s2u(bufW), 128u, 16u * n_out, SG_TILE, SG_HID, n_out);
                        umma_commit(&bar);
                    }
                    wph++;
                    mma_wait(&bar, ph & 1u, a.mma_ns, ok);
                    ph++;
                    tc_after_sync();
                    if (tid == 0 && l > 1) bulk_load(bufW, a.w.WT[l - 1], SG_HID * SG_HID * 2, &bar_w);
                    float z[32];
                    tmem_ld32(lane_tm + REG + (uint32_t)c0, d);
                    tmem_ld32(lane_tm + 128u * (l - 1) + (uint32_t)c0, z);
#pragma unroll
                    for (int j = 0; j < 32; ++j) d[j] = live ? d[j] * z[j] : 0.0f;
                    tc_before_sync();
                    __syncthreads();                            // gelu'(Z_l) is read: its columns take dW
                    tc_after_sync();
                }
                const uint32_t reg = l > 0 ? 128u * (l - 1) : 0u;
                if (tid == 0) {
                    if (l == 3) gemm_issue(tm + reg, s2u(HT[3]), T_LBO, T_SBO, s2u(bufGT), T_LBO, T_SBO, SG_HID, SG_OUT, SG_TILE);   // dW^T
                    else gemm_issue(tm + reg, s2u(bufGT), T_LBO, T_SBO, s2u(HT[l]), T_LBO, T_SBO, SG_HID, n_in, SG_TILE);          // dW
                    umma_commit(&bar);
                }
                mma_wait(&bar, ph & 1u, a.mma_ns, ok);
                ph++;
                tc_after_sync();
                if (l > 0) {                                    // D and D^T are read: write the next layer's
                    __align__(16) __nv_bfloat16 h[32];
#pragma unroll
                    for (int j = 0; j < 32; ++j) h[j] = __float2bfloat16_rn(d[j]);
                    put_row(bufA, row, c0, SG_HID, h, 32);
                    put_col(bufGT, row, c0, h, 32);
                    const float w = colsum32(d, lane);
                    sdb[TRAIN ? warp & 3 : 0][c0 + lane] = w;
                }
                const int ncol = l == 3 ? SG_OUT : n_in;
                if (c0 < ncol) {
                    float v[32];
                    tmem_ld32(lane_tm + reg + (uint32_t)c0, v);
                    if (l == 3) {                               // row = input, column = output
#pragma unroll
                        for (int j = 0; j < 32; ++j)
                            if (c0 + j < SG_OUT) {
                                float* g = part + OFFW[3] + (c0 + j) * SG_HID + row;
                                *g = first ? v[j] : *g + v[j];
                            }
                    } else {                                    // row = output, column = input
                        float4* g = reinterpret_cast<float4*>(part + OFFW[l] + row * n_in + c0);
#pragma unroll
                        for (int j = 0; j < 8; ++j) {
                            float4 o = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
                            if (!first) { const float4 q = g[j]; o.x += q.x; o.y += q.y; o.z += q.z; o.w += q.w; }
                            g[j] = o;
                        }
                    }
                }
                sg_sync();
            }
        }
    }
    if (warp == 0) tmem_dealloc(tm, NCOL);
    if (!ok) atomicOr(a.err, SG_ERR_WAIT);
}

// ------------------------------------------------------------ optimiser
// the bf16 copies of weight e of layer l, in the operand layout the kernels
// bring to shared memory: W [out][in] and W^T [in][out]
__device__ __forceinline__ void put_weight(int l, int e, float p, __nv_bfloat16* W, __nv_bfloat16* WT) {
    const int n_in = l == 0 ? SG_IN : SG_HID, n_out = l == 3 ? SG_OUT : SG_HID;
    const int woff = l == 0 ? 0 : SG_HID * SG_IN + (l - 1) * SG_HID * SG_HID;      // SG_WOFF[l]
    const int o = e / n_in, in = e - o * n_in;
    const __nv_bfloat16 h = __float2bfloat16_rn(p);
    W[woff + coff(o, in, n_in) / 2] = h;
    WT[woff + coff(in, o, n_out) / 2] = h;
}
// layer of parameter i and its offset in that layer's weights, or -1 for a bias
__device__ __forceinline__ int weight_of(int i, int* e) {
    const int w0[4] = {SG_OFF_W1, SG_OFF_W2, SG_OFF_W3, SG_OFF_W4}, b0[4] = {SG_OFF_B1, SG_OFF_B2, SG_OFF_B3, SG_OFF_B4};
#pragma unroll
    for (int l = 3; l >= 0; --l)
        if (i >= w0[l]) { *e = i - w0[l]; return i < b0[l] ? l : -1; }
    return -1;
}

// the gradient: the CTAs' partial sums, added in CTA order
__device__ __forceinline__ float grad_of(const float* part, uint32_t nparts, int i) {
    float g = 0.0f;
    for (uint32_t k = 0; k < nparts; ++k) g += part[(size_t)k * SG_NPARAM + i];
    return g;
}

__global__ void k_sg_grad(const float* part, uint32_t nparts, float* g) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < SG_NPARAM) g[i] = grad_of(part, nparts, i);
}

__global__ void k_sg_adam(float* p, float* m, float* v, const float* part, uint32_t nparts, float lr, float b1t, float b2t,
                          __nv_bfloat16* W, __nv_bfloat16* WT) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= SG_NPARAM) return;
    const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    const float gi = grad_of(part, nparts, i);
    const float mi = b1 * m[i] + (1.0f - b1) * gi;
    const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
    m[i] = mi; v[i] = vi;
    const float mh = mi / (1.0f - b1t), vh = vi / (1.0f - b2t);
    const float pi = p[i] - lr * mh / (sqrtf(vh) + eps);
    p[i] = pi;
    int e = 0;
    const int l = weight_of(i, &e);
    if (l >= 0) put_weight(l, e, pi, W, WT);
}

__global__ void k_sg_convert(const float* p, __nv_bfloat16* W, __nv_bfloat16* WT) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= SG_NPARAM) return;
    int e = 0;
    const int l = weight_of(i, &e);
    if (l >= 0) put_weight(l, e, p[i], W, WT);
}

__global__ void k_sg_standardise(const float* in, float* out, uint64_t n, int dim, const float* mean,
                                 const float* inv_std) {
    const uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (i >= n * dim) return;
    const int k = (int)(i % dim);
    out[i] = (in[i] - mean[k]) * inv_std[k];
}

// ------------------------------------------------------------ descriptors
// Per track, from its rad_buf entries in canonical order:
//   0..5   yields per 100 eV of OH, e-aq (codes 1 and 5), H, H3O+, OH-, H2 markers
//   6, 7   log10 E, log10 entries
//   8      log10 radius of gyration (nm)
//   9..24  histogram of log10 |x_i - x_{i-1}| between consecutive entries (16 bins, 0.01-100 nm)
//   25..40 the same for |x_i - x_{i-4}|
//   41..56 the same for |x_i - x_{i-16}|
//   57..62 species fractions of the same six classes
//   63     1
__device__ __forceinline__ int dbin(float d) {
    const float t = (log10f(fmaxf(d, 1e-6f)) + 2.0f) * 4.0f;
    return t < 0.0f ? 0 : t >= 15.0f ? 15 : (int)t;
}

// dbin(sqrtf(d2)) by table: the bins' edges are 1.66 octaves of d2 apart, so an
// octave holds at most one.  DBIN_N octaves from 2^-12 on: the bin at the
// octave's start and the d2 from which the next one holds.  The edges are those of
// dbin itself, found by bisection over the f32 values (k_dbin_table, once per
// network); the two agree on every non-negative finite f32 d2 (compared one by
// one on the device).
constexpr int DBIN_N = SG_DBIN, DBIN_E0 = 127 - 12;
__global__ void k_dbin_table(float2* tab) {
    __shared__ uint32_t edge[16];
    if (threadIdx.x < 16) {
        uint32_t lo = 0, hi = 0x7f7fffffu;            // edge in (lo, hi] for bins 1..15
        while (hi - lo > 1) {
            const uint32_t mid = lo + (hi - lo) / 2;
            if (dbin(sqrtf(__uint_as_float(mid))) >= (int)threadIdx.x) hi = mid; else lo = mid;
        }
        edge[threadIdx.x] = threadIdx.x ? hi : 0u;
    }
    __syncthreads();
    if (threadIdx.x < DBIN_N) {
        const uint32_t b0 = (DBIN_E0 + threadIdx.x) << 23;
        int k = 0;
        while (k < 15 && edge[k + 1] <= b0) ++k;
        // (no d2 is at or above a NaN: the last bin holds infinity too)
        tab[threadIdx.x] = make_float2(__uint_as_float(k < 15 ? edge[k + 1] : 0x7fffffffu), __int_as_float(k));
    }
}

// What bounds it: 16 bytes per entry, read once from HBM; on the way there, the
// instructions per entry (three distances to earlier entries, which hit L1).  Bins
// come from the table instead of log10f and sqrtf, and are counted in u32 (a shared
// f32 add is a compare-and-swap loop).  One warp per track, so that the f64 sums of
// the gyration radius keep one order.
// Measured at 4096 x 10 keV: 173 us with log10f and f32 counters, 50 us now.
__global__ void __launch_bounds__(128) k_descriptors(DescArgs a) {
    __shared__ uint32_t sh[4][48];
    __shared__ float2 tab[DBIN_N];
    const int lane = threadIdx.x & 31, wl = threadIdx.x >> 5;
    if (threadIdx.x < DBIN_N) tab[threadIdx.x] = a.dbin[threadIdx.x];
    __syncthreads();
    uint32_t* h = sh[wl];
    for (uint32_t p = blockIdx.x * 4 + wl; p < a.nseg; p += gridDim.x * 4) {
        for (int k = lane; k < 48; k += 32) h[k] = 0u;
        __syncwarp();
        const unsigned long long s = a.seg_off[p], e = a.seg_off[p + 1];
        const uint32_t n = (uint32_t)(e - s);
        const float4* R = a.rad + s;
        double sx = 0, sy = 0, sz = 0, s2 = 0;
        uint32_t cls[6] = {0, 0, 0, 0, 0, 0};
        auto entry = [&](uint32_t i, const float4& q, const float4* o) {
            const int code = (int)rintf(q.w) % 8;
            const int k = code == 0 ? 0 : (code == 1 || code == 5) ? 1 : code == 2 ? 2 : code == 3 ? 3
                        : code == 6 ? 4 : 5;
#pragma unroll
            for (int c = 0; c < 6; ++c) cls[c] += k == c;
            sx += q.x; sy += q.y; sz += q.z;
            s2 += (double)q.x * q.x + (double)q.y * q.y + (double)q.z * q.z;
#pragma unroll
            for (int t = 0; t < 3; ++t) {
                if (i < (t == 0 ? 1u : t == 1 ? 4u : 16u)) continue;
                const float dx = q.x - o[t].x, dy = q.y - o[t].y, dz = q.z - o[t].z;
                const float d2 = fmaxf(dx * dx + dy * dy + dz * dz, 0.0f);       // a NaN counts as 0, as in dbin
                const int oct = min(max((int)(__float_as_uint(d2) >> 23) - DBIN_E0, 0), DBIN_N - 1);
                const float2 b = tab[oct];
                atomicAdd(&h[16 * t + __float_as_int(b.y) + (d2 >= b.x ? 1 : 0)], 1u);
            }
        };
        // two entries per lane and turn: their eight loads are in flight together
        for (uint32_t i = lane; i < n; i += 64) {
            const uint32_t j = i + 32;
            const bool two = j < n;
            const uint32_t j2 = two ? j : i;
            const float4 q0 = R[i], q1 = R[j2];
            const float4 o0[3] = {R[i >= 1 ? i - 1 : 0], R[i >= 4 ? i - 4 : 0], R[i >= 16 ? i - 16 : 0]};
            const float4 o1[3] = {R[j2 >= 1 ? j2 - 1 : 0], R[j2 >= 4 ? j2 - 4 : 0], R[j2 >= 16 ? j2 - 16 : 0]};
            entry(i, q0, o0);
            if (two) entry(j, q1, o1);
        }
        for (int o = 16; o; o >>= 1) {
            sx += __shfl_xor_sync(0xffffffffu, sx, o); sy += __shfl_xor_sync(0xffffffffu, sy, o);
            sz += __shfl_xor_sync(0xffffffffu, sz, o); s2 += __shfl_xor_sync(0xffffffffu, s2, o);
#pragma unroll
            for (int k = 0; k < 6; ++k) cls[k] += __shfl_xor_sync(0xffffffffu, cls[k], o);
        }
        __syncwarp();
        const float E = a.E ? a.E[p] : a.E0;
        float* out = a.out + (size_t)p * 64;
        if (lane == 0) {
            const float per100 = E > 0 ? E / 100.0f : 1.0f;
#pragma unroll
            for (int k = 0; k < 6; ++k) {
                out[k] = (float)cls[k] / per100;
                out[57 + k] = n ? (float)cls[k] / (float)n : 0.0f;
            }
            out[6] = log10f(fmaxf(E, 1.0f));
            out[7] = log10f((float)n + 1.0f);
            double rg2 = 0.0;
            if (n) {
                const double cx = sx / n, cy = sy / n, cz = sz / n;
                rg2 = s2 / n - (cx * cx + cy * cy + cz * cz);
            }
            out[8] = log10f((float)sqrt(fmax(rg2, 0.0)) + 0.01f);
            out[63] = 1.0f;
        }
#pragma unroll
        for (int t = 0; t < 3; ++t) {
            const uint32_t L = t == 0 ? 1 : t == 1 ? 4 : 16;
            const float norm = n > L ? 1.0f / (float)(n - L) : 0.0f;
            if (lane < 16) out[9 + 16 * t + lane] = (float)h[16 * t + lane] * norm;
        }
        __syncwarp();
    }
}

// ------------------------------------------------------------ launchers
static int sm_count() {
    int dev = 0, n = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    return n > 0 ? n : 148;
}

cudaError_t launch_dbin_table(float2* tab, cudaStream_t s) {
    k_dbin_table<<<1, 32, 0, s>>>(tab);
    return cudaGetLastError();
}

cudaError_t launch_descriptors(const DescArgs& a, cudaStream_t s) {
    if (a.nseg == 0) return cudaSuccess;
    const uint32_t want = (a.nseg + 3) / 4, cap = (uint32_t)sm_count() * 8;
    const int blocks = (int)(want < cap ? want : cap);
    k_descriptors<<<blocks, 128, 0, s>>>(a);
    return cudaGetLastError();
}

static uint32_t sg_tiles(uint32_t n) { return (n + SG_TILE - 1) / SG_TILE; }

cudaError_t launch_sg_forward(const SgArgs& a, cudaStream_t s) {
    if (a.n == 0) return cudaSuccess;
    static DeviceOnce attr;
    cudaError_t e = attr.run([] {
        return cudaFuncSetAttribute(k_sg<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SG_SMEM_FWD);
    });
    if (e != cudaSuccess) return e;
    k_sg<false><<<sg_tiles(a.n), SG_THREADS, SG_SMEM_FWD, s>>>(a);
    return cudaGetLastError();
}

uint32_t sg_parts(uint32_t n) {
    const uint32_t t = sg_tiles(n), c = (uint32_t)sm_count();
    return t < c ? t : c;
}

cudaError_t launch_sg_train(const SgArgs& a, cudaStream_t s) {
    if (a.n == 0) return cudaSuccess;
    static DeviceOnce attr;
    cudaError_t e = attr.run([] {
        return cudaFuncSetAttribute(k_sg<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SG_SMEM_TRAIN);
    });
    if (e != cudaSuccess) return e;
    k_sg<true><<<sg_parts(a.n), SG_THREADS, SG_SMEM_TRAIN, s>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_sg_adam(float* p, float* m, float* v, const float* part, uint32_t nparts, float lr, float b1t,
                           float b2t, __nv_bfloat16* Wcat, __nv_bfloat16* WTcat, cudaStream_t s) {
    k_sg_adam<<<(SG_NPARAM + 255) / 256, 256, 0, s>>>(p, m, v, part, nparts, lr, b1t, b2t, Wcat, WTcat);
    return cudaGetLastError();
}

cudaError_t launch_sg_grad(const float* part, uint32_t nparts, float* g, cudaStream_t s) {
    k_sg_grad<<<(SG_NPARAM + 255) / 256, 256, 0, s>>>(part, nparts, g);
    return cudaGetLastError();
}

cudaError_t launch_sg_convert(const float* p, __nv_bfloat16* Wcat, __nv_bfloat16* WTcat, cudaStream_t s) {
    k_sg_convert<<<(SG_NPARAM + 255) / 256, 256, 0, s>>>(p, Wcat, WTcat);
    return cudaGetLastError();
}

cudaError_t launch_sg_standardise(const float* in, float* out, uint64_t n, int dim, const float* mean,
                                  const float* inv_std, cudaStream_t s) {
    const uint64_t tot = n * (uint64_t)dim;
    if (!tot) return cudaSuccess;
    k_sg_standardise<<<(unsigned)((tot + 255) / 256), 256, 0, s>>>(in, out, n, dim, mean, inv_std);
    return cudaGetLastError();
}

}  // namespace wg
