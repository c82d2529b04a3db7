// Internal declarations shared by the translation units of libfvm_b200 (not part of the C ABI).
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>

#include "../../include/fvm_b200.h"
#include "ptx_sm100.cuh"

namespace fvm {

struct DeviceState {
    int sms = 0;
    int max_smem = 0;
    int* status_dev = nullptr;    // device-visible address of the status word (mapped pinned host memory)
    int* status_host = nullptr;   // host address of the same word
    // stream-K scratch of the convolution kernel: fp32 partial tiles (one slot per CTA) and one counter per slot. Shared
    // by every stream of the device: stream-K launches on different streams must not overlap in time.
    float* sk_part = nullptr;
    int* sk_flags = nullptr;
    size_t sk_floats = 0;
    // completion counters of the layer-chain kernel (one per layer and 256-row tile), zeroed before every chain launch;
    // shared by every stream of the device: chain launches on different streams must not overlap in time
    int* chain_flags = nullptr;
    int chain_flag_count = 0;
    int pair_clusters = 0;        // CTA pairs (clusters of two) the device runs at once; 0: pair kernel unavailable
    bool ready = false;
};

// State of the current device, or nullptr if fvm_init() has not run for it.
DeviceState* device_state();
void count_launch();

int conv_host_init();
int conv_pair_capacity();
// cuTensorMapEncodeTiled for an fp16 tensor of `rank` dimensions (innermost first): sizes, byte strides of dimensions
// 1.., box; no interleave, swizzle of 128, 64 or 32 bytes or none (0), zero fill outside the tensor. Returns an FVM_* status.
int encode_tiled_f16(CUtensorMap* map, const void* ptr, int rank, const unsigned long long* dims,
                     const unsigned long long* strides_bytes, const unsigned* box, int swizzle_bytes);
int stem_s2_launch(const void* x, const void* w, const void* bias, void* y, int N, int H, int W, int K, int R, int S,
                   int ph, int pw, long long ldy, int act, cudaStream_t stream);
int conv2d_launch(const void* x, const void* w, const void* bias, const void* res, const float* scale, void* y, int N,
                  int H, int W, int C, int K, int R, int S, int ph, int pw, int sh, int sw, int dh, int dw,
                  long long ldx, long long ldy, long long ldr, int act, int force_bn, int ph_hi, int pw_hi,
                  cudaStream_t stream, int w_per_image = 0, int gsg = 0, int gsk = 0);
// Cluster split-K convolution (conv_split.cu): one output tile per cluster of `split` CTAs or CTA pairs.
struct SplitParams {
    int M, K, P, Q, S, sh, sw, ph, pw, dh, dw;
    int cchunks, kblocks, im2col;
    int BN, n_tiles, split;
    int pair;                          // tiles of 256 x BN, `split` CTA pairs per cluster (conv_split_pair_kernel)
    int lg_bn, stages, tmem_cols;      // from conv_split_plan
    uint32_t red_bytes;
    int act;
    int wdyn;                          // weights written by the preceding kernel: fetched after the wait for it
    const __half* bias;
    const __half* res;
    const float* scale;
    __half* y;
    long long ldy, ldr;
    FastDiv div_split, div_ntiles, div_pq, div_q;
    int* status;
};
bool conv_split_plan(SplitParams* p, size_t* smem);
int conv_split_launch(const CUtensorMap& tmap_a, const CUtensorMap& tmap_b, const SplitParams& p, size_t smem, cudaStream_t stream);
// Stride-1 7x7 depthwise convolution on the tensor cores (dwconv_mma.cu): whether a layer runs there, its squeeze slots, its
// launch.
bool dw_mma_runs(int N, int H, int W, int C, int ph, int pw);
int dw_mma_slots(int N, int H, int W, int C, int ph, int pw);
int dw_mma_launch(const void* x, const void* w, const void* bias, void* y, float* pool_partial, int N, int H, int W, int C,
                  int ph, int pw, long long ldx, long long ldy, int act, cudaStream_t stream);
int conv_chain_launch(const fvm_chain_layer* layers, int n, cudaStream_t stream);
int conv_dual_launch(const void* x, const void* w1, const void* b1, const void* res, void* y, const void* w2, const void* b2,
                     void* z, long long M, int C1, int K1, int K2, long long ldx, long long ldr, long long ldy, long long ldz,
                     int act1, int act2, cudaStream_t stream);

bool pdl_enabled();      // FVM_B200_PDL=0: plain launches
// Launch with programmatic stream serialization (the kernel calls pdl_wait before it touches activations) in clusters of
// `cluster` blocks. Measured on B200 in a replayed graph: a plain launch adds about 1 us between two small kernels.
template <typename... P, typename... A>
int launch_pdl(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, int cluster, A... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attrs[2];
    attrs[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attrs[0].val.programmaticStreamSerializationAllowed = 1;
    attrs[1].id = cudaLaunchAttributeClusterDimension;
    attrs[1].val.clusterDim.x = static_cast<unsigned>(cluster);
    attrs[1].val.clusterDim.y = 1;
    attrs[1].val.clusterDim.z = 1;
    const bool pdl = pdl_enabled();
    cfg.attrs = pdl ? attrs : attrs + 1;
    cfg.numAttrs = (pdl ? 1u : 0u) + (cluster > 1 ? 1u : 0u);
    if (cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...) != cudaSuccess) {
        (void)cudaGetLastError();
        return FVM_ERR_LAUNCH;
    }
    count_launch();
    return FVM_OK;
}

}  // namespace fvm
