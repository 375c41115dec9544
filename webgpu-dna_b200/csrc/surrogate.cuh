// surrogate.cuh -- learned chemistry: track descriptors and a 64-128-128-128-80
// GELU MLP with bf16 weights and f32 accumulation on the tcgen05 tensor cores.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>
#include <cuda_bf16.h>

namespace wg {

constexpr int SG_IN = 64, SG_HID = 128, SG_OUT = 80;
constexpr int SG_TILE = 128;                 // rows (tracks) per CTA
// f32 parameter vector: W1 [128][64], b1, W2 [128][128], b2, W3 [128][128], b3, W4 [80][128], b4
constexpr int SG_OFF_W1 = 0, SG_OFF_B1 = SG_OFF_W1 + SG_HID * SG_IN;
constexpr int SG_OFF_W2 = SG_OFF_B1 + SG_HID, SG_OFF_B2 = SG_OFF_W2 + SG_HID * SG_HID;
constexpr int SG_OFF_W3 = SG_OFF_B2 + SG_HID, SG_OFF_B3 = SG_OFF_W3 + SG_HID * SG_HID;
constexpr int SG_OFF_W4 = SG_OFF_B3 + SG_HID, SG_OFF_B4 = SG_OFF_W4 + SG_OUT * SG_HID;
constexpr int SG_NPARAM = SG_OFF_B4 + SG_OUT;

// bf16 copies of the weights, W_l [out][in] and transposed [in][out], each laid out
// as the tensor cores' K-major shared-memory operand (surrogate.cu coff)
struct SgWeights {
    const __nv_bfloat16 *W[4], *WT[4];
    const float* p;                          // f32 parameters (biases read from here)
};

struct SgArgs {
    const float* X;                          // n x 64 inputs
    const float *xmean, *xinv;               // standardise on load ((x - xmean) * xinv), or null
    const uint32_t* rows;                    // optional gather (batch -> row of X / T)
    uint32_t n;
    SgWeights w;
    uint32_t* err;
    unsigned long long mma_ns;               // bound of a tensor-core or bulk-copy wait
    uint32_t give_up_first;                  // test switch: a tile's first wait gives up at once
    // forward: outputs y * ystd + ymean to Y (n x 80, may be null), and / or their
    // energy-weighted sums ((y * ystd + ymean) * E_track, then E_track) added to acc[0..80]
    float* Y;
    const float *ymean, *ystd;
    const float* E;                          // per-row energy, or null for E0
    float E0;
    double* acc;
    // training: targets (standardised, gathered like X), the CTAs' partial gradients
    // (sg_parts(n) x SG_NPARAM, overwritten) and the sum of squared errors (added to)
    const float* T;
    float* part;
    double* loss;
};

// descriptors of the tracks of a canonical rad_buf
struct DescArgs {
    const float4* rad;
    const unsigned long long* seg_off;
    uint32_t nseg;
    const float* E;                          // per-track energy (eV) or null
    float E0;                                // energy when E is null
    float* out;                              // nseg x 64
    const float2* dbin;                      // the distance bins' table (launch_dbin_table)
};

// the table of the descriptors' distance bins, SG_DBIN entries
constexpr int SG_DBIN = 25;
cudaError_t launch_dbin_table(float2* tab, cudaStream_t s);
cudaError_t launch_descriptors(const DescArgs& a, cudaStream_t s);
cudaError_t launch_sg_forward(const SgArgs& a, cudaStream_t s);
// loss and partial gradients of n rows, by sg_parts(n) CTAs of the current device
cudaError_t launch_sg_train(const SgArgs& a, cudaStream_t s);
uint32_t sg_parts(uint32_t n);
// Adam on the f32 parameters with the sum of the partial gradients, then the bf16 weight copies
cudaError_t launch_sg_adam(float* p, float* m, float* v, const float* part, uint32_t nparts, float lr, float b1t,
                           float b2t, __nv_bfloat16* Wcat, __nv_bfloat16* WTcat, cudaStream_t s);
// that sum alone
cudaError_t launch_sg_grad(const float* part, uint32_t nparts, float* g, cudaStream_t s);
// bf16 copies of the weights only
cudaError_t launch_sg_convert(const float* p, __nv_bfloat16* Wcat, __nv_bfloat16* WTcat, cudaStream_t s);
// standardise rows: out = (in - mean) / std
cudaError_t launch_sg_standardise(const float* in, float* out, uint64_t n, int dim, const float* mean,
                                  const float* inv_std, cudaStream_t s);
// offsets of W_l (and WT_l) inside the concatenated bf16 arrays
constexpr int SG_WOFF[4] = {0, SG_HID * SG_IN, SG_HID * SG_IN + SG_HID * SG_HID, SG_HID * SG_IN + 2 * SG_HID * SG_HID};
constexpr int SG_WTOTAL = SG_HID * SG_IN + 2 * SG_HID * SG_HID + SG_OUT * SG_HID;

}  // namespace wg
